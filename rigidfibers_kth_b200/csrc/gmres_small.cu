// gmres_small.cu - the whole FP64 GMRES(m) solve of a small system in one
// cooperative kernel.
//
// The flow is the one of gmres.h (fortran/dGMRES.f:491-1495): warm start, CGS2
// orthogonalisation as in arnoldi.cu, Givens rotations, the true residual when
// the estimate meets the tolerance; a restart takes its residual from the
// cycle's basis, as there.  What bounds a small system is the chain of
// launches: a step of the device-controlled solver is six kernels, 31 us at n =
// 1500 where the product reads its 18 MB from L2 in about 3.  Here a step's phases are separated by two grid barriers:
//   product    a CTA's own rows (up to kSmallRows) of A v, kept in its shared
//              memory with its rows of the basis, of the basis' products and
//              of x; partial dot products h1 = V^T w;
//   w -= V h1  goes out to all; partial dot products h2 = V^T w and |w|^2.
// The second correction, w - V h2, stays at home: its norm is |w|^2 - |h2|^2
// (h2 is rounding), the next product is made with the vector that went out and
// corrected by (A V) h2, which the CTA has for its rows.  Where the difference
// cancels by more than half, w - V h2 goes out and its norm takes a barrier of
// its own.  The barrier is the cost of a small system, some 2.5 us with the
// sums behind it: a product split over all warps of the grid with its partial
// sums behind a barrier, and |w| behind another, took 14.1 us a step at n =
// 1500 (four barriers) where this takes 12.5.  A barrier made of the sums
// themselves (tagged 16-byte values that every warp polls) took 19: the polls
// hold up the values they wait for.
// Every CTA adds the CTAs' partial sums in the same order and carries its own
// copy of the Hessenberg matrix, the rotations and the stop test, so that all
// take the same decisions without another exchange.  A barrier that waits too
// long sets an error and the CTAs leave.
//
// Device-controlled passes -> this kernel, a step to 1e-10: n = 1500 31 -> 12.5
// us, n = 3000 44 -> 17 us, n = 4500 (162 MB, from memory) 58 -> 34 us.
// Systems up to kSmallMaxN = 8192: there the product of 537 MB takes 80 of the
// 90 us a step costs here, and the passes' launches hide behind it from about
// there on; a CTA's rows (kSmallRows = 64 on each SM) end at 9472.
#include <algorithm>
#include <cmath>

#include "rf_kernels.h"

namespace rf {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int KM = kArnoldiMax;
static_assert(kWarps >= KM, "a warp per basis vector");
constexpr int kSumLoads = 5;                         // 160 CTAs in one round
constexpr long long kWaitLimit = 4000000000;    // cycles: some two seconds

struct Shared {
    double V[KM][kSmallRows], AV[KM][kSmallRows];  // the basis and its products
    double w[kSmallRows], x[kSmallRows], xcur[kSmallRows], b[kSmallRows];
    double red[kWarps * 4 * (16 + 1)];             // the warps' partial sums: 16 cols x (2 half + 1)
    double h1[KM], h2[KM + 1];                     // h2[j + 1] = |w|^2
    double H[KM][KM], g[KM + 1], cs[KM], sn[KM], y[KM + 1];
    double sum[2];
    int failed;
};

__device__ void rotg(double a, double b, double *c, double *s) {  // LINPACK drotg (fortran/blas_rot.f:117-146)
    const double roe = (fabs(a) > fabs(b)) ? a : b;
    const double scale = fabs(a) + fabs(b);
    if (scale == 0.0) {
        *c = 1.0;
        *s = 0.0;
        return;
    }
    double r = scale * sqrt((a / scale) * (a / scale) + (b / scale) * (b / scale));
    r = copysign(1.0, roe) * r;
    *c = a / r;
    *s = b / r;
}

__device__ __forceinline__ void rot(double &x, double &y, double c, double s) {
    const double t = c * x + s * y;
    y = c * y - s * x;
    x = t;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

struct Solver {
    const SmallGmresArgs &a;
    Shared &s;
    int r0, rows;            // this CTA's rows
    int half, cols;          // lanes of a column, columns a warp reads at once
    unsigned phase = 0;      // barriers passed

    template <int B, int COLS>
    __device__ __forceinline__ void batch(const double *q, int c, int g, bool act, double xl, double &s0,
                                          double &s1) const {
        double2 t[B];
#pragma unroll
        for (int e = 0; e < B; ++e)
            t[e] = act ? __ldg(reinterpret_cast<const double2 *>(q + (int64_t)(c + e * COLS) * a.lda))
                       : make_double2(0.0, 0.0);
#pragma unroll
        for (int e = 0; e < B; ++e) {
            const double xv = __shfl_sync(0xffffffffu, xl, (c + e * COLS + g) & 31);
            s0 = fma(t[e].x, xv, s0);
            s1 = fma(t[e].y, xv, s1);
        }
    }

    // s.w = this CTA's rows of A (scale v), or of b less it.  A column's rows are
    // read by `half` lanes, two rows each; the warps stride over the columns, 32
    // at a time, `cols` of them at once.
    __device__ void product(const double *v, double scale, bool residual) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int g = lane / half, l = lane - g * half, n = (int)a.n, ld = 2 * half + 1;
        const bool act = g < cols && 2 * l < rows;
        const double *p = a.A + r0 + 2 * l + (int64_t)g * a.lda;
        double s0 = 0.0, s1 = 0.0;
        if (rows > 0)
            for (int cb = warp * 32; cb < n; cb += kWarps * 32) {
                const double xl = cb + lane < n ? scale * __ldcg(v + cb + lane) : 0.0;
                const double *q = p + (int64_t)cb * a.lda;
                const int nc = min(32, n - cb);
                int c = 0;
                if (cols == 4)
                    for (; c + 32 <= nc; c += 32) batch<8, 4>(q, c, g, act, xl, s0, s1);
                else if (cols == 2)
                    for (; c + 16 <= nc; c += 16) batch<8, 2>(q, c, g, act, xl, s0, s1);
                else
                    for (; c + 16 <= nc; c += 16) batch<16, 1>(q, c, g, act, xl, s0, s1);
                for (; c < nc; c += cols) {
                    const double xv = __shfl_sync(0xffffffffu, xl, (c + g) & 31);
                    if (act && c + g < nc) {
                        const double2 t = __ldg(reinterpret_cast<const double2 *>(q + (int64_t)c * a.lda));
                        s0 = fma(t.x, xv, s0);
                        s1 = fma(t.y, xv, s1);
                    }
                }
            }
        if (act) {
            double *o = s.red + (warp * cols + g) * ld + 2 * l;
            o[0] = s0;
            o[1] = s1;
        }
        __syncthreads();
        // eight threads a row
        const int r = threadIdx.x >> 3;
        double t = 0.0;
        if (r < rows)
            for (int u = threadIdx.x & 7; u < kWarps * cols; u += 8) t += s.red[u * ld + r];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (r < rows && (threadIdx.x & 7) == 0) s.w[r] = residual ? s.b[r] - t : t;
        __syncthreads();
    }

    // every CTA's writes before, every CTA's reads after; false: gave up
    __device__ bool barrier() {
        __syncthreads();
        ++phase;
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.barrier) : "memory");
            const unsigned target = phase * gridDim.x;
            const long long t0 = clock64();
            while (true) {
                unsigned v;
                asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(v) : "l"(a.barrier) : "memory");
                if ((int)(v - target) >= 0) break;
                if (clock64() - t0 > kWaitLimit) {
                    s.failed = 1;
                    // the host looks here too: the CTA that came last may pass, and
                    // the first CTA finish the solve, without this one's rows
                    *static_cast<volatile unsigned *>(a.barrier + 1) = 1;
                    break;
                }
            }
        }
        __syncthreads();
        return !s.failed;
    }

    // out[q] = sum over the grid of u . v over the CTAs' rows, q < cnt <= KM + 1,
    // a warp per q.  The places alternate between two sets: a CTA that writes
    // one again has passed the barrier that all CTAs reach only after reading it.
    template <typename F>
    __device__ bool dots(int cnt, F value, double *out) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        double *set = a.sums + (int64_t)(phase & 1) * (KM + 1) * gridDim.x;
        for (int q = warp; q < cnt; q += kWarps) {
            double t = 0.0;
            for (int r = lane; r < rows; r += 32) t += value(q, r);
            t = warp_sum(t);
            if (lane == 0) set[q * gridDim.x + blockIdx.x] = t;
        }
        if (!barrier()) return false;
        for (int q = warp; q < cnt; q += kWarps) {
            double t = 0.0;
            for (int b0 = lane; b0 < (int)gridDim.x; b0 += 32 * kSumLoads) {
                double v[kSumLoads];  // all in flight together: one trip to L2
#pragma unroll
                for (int e = 0; e < kSumLoads; ++e)
                    v[e] = b0 + 32 * e < (int)gridDim.x ? __ldcg(set + q * gridDim.x + b0 + 32 * e) : 0.0;
#pragma unroll
                for (int e = 0; e < kSumLoads; ++e) t += v[e];
            }
            t = warp_sum(t);
            if (lane == 0) out[q] = t;
        }
        __syncthreads();
        return true;
    }

    // this CTA's rows of a vector in shared memory, to global memory
    __device__ void publish(double *dst, const double *src) const {
        for (int r = threadIdx.x; r < rows; r += kThreads) dst[r0 + r] = src[r];
    }

    // s.w = b - A x for x in global memory, its norm; false: gave up
    __device__ bool residual(const double *x, double *norm) {
        product(x, 1.0, true);
        publish(a.w, s.w);
        if (!dots(1, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return false;
        *norm = sqrt(s.sum[0]);
        return true;
    }

    // s.xcur = s.x + V y, y from the k steps done
    __device__ void combine(int k) {
        if (threadIdx.x == 0) {
            for (int r = 0; r < k; ++r) s.y[r] = s.g[r];
            for (int c = k - 1; c >= 0; --c) {
                s.y[c] /= s.H[c][c];
                for (int r = 0; r < c; ++r) s.y[r] -= s.y[c] * s.H[c][r];
            }
        }
        __syncthreads();
        for (int r = threadIdx.x; r < rows; r += kThreads) {
            double t = 0.0;
            for (int q = 0; q < k; ++q) t += s.V[q][r] * s.y[q];
            s.xcur[r] = s.x[r] + t;
        }
        __syncthreads();
    }

    __device__ void run() {
        SmallGmresStat st{};
        auto leave = [&](int info) {
            st.info = info;
            if (blockIdx.x == 0 && threadIdx.x == 0) *a.stat = st;
        };
        if (threadIdx.x == 0) s.failed = 0;
        for (int r = threadIdx.x; r < rows; r += kThreads) {
            s.x[r] = a.x[r0 + r];
            s.b[r] = a.b[r0 + r];
        }
        // without a right-hand side (one fiber, or no external force) x = 0; every
        // CTA looks at all of b, as no barrier costs less
        bool any = false;
        for (int r = threadIdx.x; r < (int)a.n; r += kThreads) any = any || a.b[r] != 0.0;
        if (!__syncthreads_or(any)) {
            for (int r = threadIdx.x; r < rows; r += kThreads) a.x[r0 + r] = 0.0;
            return leave(kSmallOk);
        }
        product(a.x, 1.0, true);
        ++st.matvecs;
        publish(a.w, s.w);
        if (!dots(2, [&](int q, int r) { return q == 0 ? s.b[r] * s.b[r] : s.w[r] * s.w[r]; }, s.sum))
            return leave(kSmallTimeout);
        const double bn = sqrt(s.sum[0]);
        double beta = sqrt(s.sum[1]);
        if (!isfinite(bn)) return leave(kSmallNaN);
        if (bn == 0.0) {
            for (int r = threadIdx.x; r < rows; r += kThreads) a.x[r0 + r] = 0.0;
            return leave(kSmallOk);
        }
        if (!isfinite(beta)) return leave(kSmallNaN);
        if (beta == 0.0) return leave(kSmallOk);
        bool check_failed = false;  // an estimate within the tolerance whose true residual was not
        for (;;) {
            double norm = beta;  // of the vector in s.w
            bool ahead = false;  // a.w is that vector before its second correction (by V h2)
            if (threadIdx.x <= KM) s.g[threadIdx.x] = threadIdx.x == 0 ? beta : 0.0;
            double bea = 0.0;
            bool stopped = false;  // xcur holds the estimate's solution
            for (int j = 0; j < a.m; ++j) {
                const double inv = 1.0 / norm;
                for (int r = threadIdx.x; r < rows; r += kThreads) s.V[j][r] = s.w[r] * inv;
                product(a.w, inv, false);
                ++st.matvecs;
                // where a.w is the vector before its second correction, the
                // product is corrected: A (w - V h2) = A w - (A V) h2
                for (int r = threadIdx.x; r < rows; r += kThreads) {
                    double t = s.w[r];
                    if (ahead)
                        for (int q = 0; q < j; ++q) t -= s.h2[q] * inv * s.AV[q][r];
                    s.w[r] = s.AV[j][r] = t;
                }
                __syncthreads();
                if (!dots(j + 1, [&](int q, int r) { return s.V[q][r] * s.w[r]; }, s.h1)) return leave(kSmallTimeout);
                for (int r = threadIdx.x; r < rows; r += kThreads) {
                    double t = s.w[r];
                    for (int q = 0; q <= j; ++q) t -= s.h1[q] * s.V[q][r];
                    s.w[r] = t;
                    a.w[r0 + r] = t;
                }
                __syncthreads();
                if (!dots(j + 2, [&](int q, int r) { return (q <= j ? s.V[q][r] : s.w[r]) * s.w[r]; }, s.h2))
                    return leave(kSmallTimeout);
                // |w - V h2|^2 = |w|^2 - |h2|^2, unless that cancels
                const double ww = s.h2[j + 1];
                double left = ww;
                for (int q = 0; q <= j; ++q) left -= s.h2[q] * s.h2[q];
                ahead = left > 0.5 * ww;
                for (int r = threadIdx.x; r < rows; r += kThreads) {
                    double t = s.w[r];
                    for (int q = 0; q <= j; ++q) t -= s.h2[q] * s.V[q][r];
                    s.w[r] = t;
                    if (!ahead) a.w[r0 + r] = t;
                }
                __syncthreads();
                if (ahead) {
                    norm = sqrt(left);
                } else {
                    if (!dots(1, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return leave(kSmallTimeout);
                    norm = sqrt(s.sum[0]);
                }
                if (threadIdx.x == 0) {
                    // column j: the earlier rotations as one chain over x, the
                    // loads of the next ones ahead of it
                    double *h = s.H[j];
                    bool finite = isfinite(norm);
                    double x = s.h1[0] + s.h2[0];
                    finite = finite && isfinite(x);
                    for (int r = 0; r < j; r += 4) {
                        double y[4], c[4], sn[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (r + e < j) {
                                y[e] = s.h1[r + e + 1] + s.h2[r + e + 1];
                                c[e] = s.cs[r + e];
                                sn[e] = s.sn[r + e];
                            }
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (r + e < j) {
                                finite = finite && isfinite(y[e]);
                                rot(x, y[e], c[e], sn[e]);
                                h[r + e] = x;
                                x = y[e];
                            }
                    }
                    h[j] = x;
                    double hn = norm;
                    rotg(h[j], hn, &s.cs[j], &s.sn[j]);
                    rot(s.g[j], s.g[j + 1], s.cs[j], s.sn[j]);
                    rot(h[j], hn, s.cs[j], s.sn[j]);
                    s.sum[1] = finite ? fabs(s.g[j + 1]) / bn : nan("");
                }
                __syncthreads();
                bea = s.sum[1];
                ++st.iterations;
                st.backward_error = bea;
                if (!isfinite(bea)) return leave(kSmallNaN);
                stopped = bea <= a.tol || st.iterations >= a.max_iters;
                if (!stopped) continue;
                // the true residual decides
                combine(j + 1);
                publish(a.xcur, s.xcur);
                // s.w and a.w hold the next basis vector: the residual must not
                // take their place while the cycle may go on
                for (int r = threadIdx.x; r < rows; r += kThreads) s.V[KM - 1][r] = j + 1 < KM ? s.w[r] : 0.0;
                if (!barrier()) return leave(kSmallTimeout);
                product(a.xcur, 1.0, true);
                ++st.matvecs;
                if (!dots(1, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return leave(kSmallTimeout);
                st.backward_error = sqrt(s.sum[0]) / bn;
                if (st.backward_error <= a.tol || st.iterations >= a.max_iters) {
                    publish(a.x, s.xcur);
                    return leave(st.backward_error <= a.tol ? kSmallOk : kSmallBudget);
                }
                for (int r = threadIdx.x; r < rows; r += kThreads) s.w[r] = j + 1 < KM ? s.V[KM - 1][r] : 0.0;
                __syncthreads();
                check_failed = true;
            }
            // restart from the residual of the updated x, without a product
            // where the cycle's basis may give it (arnoldi.cu)
            if (!stopped) combine(a.m);
            for (int r = threadIdx.x; r < rows; r += kThreads) s.x[r] = s.xcur[r];
            if (check_failed) {
                publish(a.xcur, s.xcur);
                if (!barrier()) return leave(kSmallTimeout);
                ++st.matvecs;
                if (!residual(a.xcur, &beta)) return leave(kSmallTimeout);
            } else {
                if (threadIdx.x == 0) {
                    double t = s.g[a.m];
                    for (int q = a.m - 1; q >= 0; --q) {
                        s.y[q + 1] = s.cs[q] * t;
                        t *= -s.sn[q];
                    }
                    s.y[0] = t;
                    s.y[a.m] /= norm;
                }
                __syncthreads();
                for (int r = threadIdx.x; r < rows; r += kThreads) {
                    double t = s.y[a.m] * s.w[r];
                    for (int q = 0; q < a.m; ++q) t += s.y[q] * s.V[q][r];
                    s.w[r] = t;
                    a.w[r0 + r] = t;
                }
                __syncthreads();
                if (!dots(1, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return leave(kSmallTimeout);
                beta = sqrt(s.sum[0]);
            }
            if (!isfinite(beta)) return leave(kSmallNaN);
            if (beta == 0.0) {
                publish(a.x, s.x);
                st.backward_error = 0.0;
                return leave(kSmallOk);
            }
        }
    }
};

__global__ void __launch_bounds__(kThreads, 1) gmres_small_kernel(SmallGmresArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    Shared &s = *reinterpret_cast<Shared *>(smem);
    // four rows are a whole 32-byte sector of a column
    const int per = (int)((a.n + gridDim.x - 1) / gridDim.x + 3) / 4 * 4, half = per / 2;
    const int r0 = min((int)a.n, (int)blockIdx.x * per), r1 = min((int)a.n, r0 + per);
    Solver v{a, s, r0, r1 - r0, half, half <= 8 ? 4 : half <= 16 ? 2 : 1};
    v.run();
}

}  // namespace

bool gmres_small_supported(int64_t n, int m, int sm_count) {
    return n >= 1 && m >= 1 && m <= KM && n <= kSmallMaxN && (n + sm_count - 1) / sm_count <= kSmallRows;
}

// two sets of sums, w, xcur
int64_t gmres_small_work(int64_t n, int sm_count) { return 2LL * (KM + 1) * sm_count + 2 * n; }

cudaError_t launch_gmres_small(SmallGmresArgs a, double *work, int sm_count, cudaStream_t st) {
    a.sums = work;
    a.w = work + 2LL * (KM + 1) * sm_count;
    a.xcur = a.w + a.n;
    cudaError_t e = cudaFuncSetAttribute(gmres_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(Shared));
    if (e == cudaSuccess) e = cudaMemsetAsync(a.barrier, 0, 2 * sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel(reinterpret_cast<void *>(gmres_small_kernel), dim3(sm_count), dim3(kThreads), args,
                                       sizeof(Shared), st);
}

}  // namespace rf
