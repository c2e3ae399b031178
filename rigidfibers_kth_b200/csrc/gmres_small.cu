// gmres_small.cu - the whole FP64 GMRES(m) solve of a small system in one
// cooperative kernel.
//
// The flow is the one of gmres.h (fortran/dGMRES.f:491-1495): warm start, CGS2
// orthogonalisation as in arnoldi.cu, Givens rotations, the true residual when
// the estimate meets the tolerance and at each restart.  What bounds a small
// system is the chain of launches: a step of the device-controlled solver is
// six kernels, 36 us at n = 1500 where the product reads its 18 MB from L2 in
// about 3.  Here the steps' phases are separated by grid barriers, four per
// step:
//   product    a warp owns 64 rows x a range of columns of A; partial sums;
//   h1 = V^T w each CTA adds the partial sums of its own rows (up to
//              kSmallRows) and keeps them, its rows of the basis and of x in
//              shared memory; partial dot products;
//   h2 = V^T w after w -= V h1;
//   |w|        after w -= V h2; w goes out unscaled, and the next product
//              scales it by 1 / |w|.
// Every CTA adds the CTAs' partial sums in the same order and carries its own
// copy of the Hessenberg matrix, the rotations and the stop test, so that all
// take the same decisions without another exchange.  A barrier that waits too
// long sets an error and the CTAs leave.
//
// Whole solves to 1e-10, device-controlled passes -> this kernel: M = 100 (n =
// 1500, 18 iterations) 0.66 -> 0.30 ms, n = 2997 0.89 -> 0.40 ms, n = 4500 (162
// MB, from memory) 58 -> 39 us an iteration.  Systems up to kSmallMaxN = 8192:
// there the product of 537 MB takes 80 of the 93 us an iteration costs here,
// and the passes' launches hide behind it from about there on; a CTA's rows
// (kSmallRows = 64 on each SM) end at 9472.
#include <algorithm>
#include <cmath>

#include "rf_kernels.h"

namespace rf {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int KM = kArnoldiMax;
static_assert(kWarps >= KM, "a warp per basis vector");
constexpr int kTileRows = 64;                      // rows of a warp's part of the product
constexpr long long kBarrierLimit = 4000000000;    // cycles: some two seconds

struct Shared {
    double V[KM][kSmallRows];
    double w[kSmallRows], x[kSmallRows], xcur[kSmallRows], b[kSmallRows];
    double red[kThreads / 16][kSmallRows + 1];     // slices of a row's partial sums
    double h1[KM], h2[KM];
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
    unsigned phase = 0;      // barriers passed

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
                if (clock64() - t0 > kBarrierLimit) {
                    s.failed = 1;
                    break;
                }
            }
        }
        __syncthreads();
        return !s.failed;
    }

    // partial sums of A (scale v) over the warps' parts
    __device__ void product(const double *v, double scale) const {
        const int lane = threadIdx.x & 31;
        const int u = blockIdx.x * kWarps + (threadIdx.x >> 5);
        if (u >= a.tiles * a.splits) return;
        const int split = u / a.tiles, tile = u - split * a.tiles;
        const int64_t row = (int64_t)tile * kTileRows + 2 * lane;
        const int c0 = split * a.cols, c1 = min((int)a.n, c0 + a.cols);
        const double *p = a.A + (int64_t)c0 * a.lda + row;
        double s0 = 0.0, s1 = 0.0;
        for (int cb = c0; cb < c1; cb += 32) {
            const double xl = cb + lane < c1 ? scale * __ldcg(v + cb + lane) : 0.0;
            const int nc = min(32, c1 - cb);
            int c = 0;
            for (; c + 8 <= nc; c += 8) {
                double2 t[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) t[e] = __ldg(reinterpret_cast<const double2 *>(p + (int64_t)e * a.lda));
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const double xv = __shfl_sync(0xffffffffu, xl, c + e);
                    s0 = fma(t[e].x, xv, s0);
                    s1 = fma(t[e].y, xv, s1);
                }
                p += 8 * a.lda;
            }
            for (; c < nc; ++c, p += a.lda) {
                const double2 t = __ldg(reinterpret_cast<const double2 *>(p));
                const double xv = __shfl_sync(0xffffffffu, xl, c);
                s0 = fma(t.x, xv, s0);
                s1 = fma(t.y, xv, s1);
            }
        }
        *reinterpret_cast<double2 *>(a.part + (int64_t)split * a.tiles * kTileRows + row) = make_double2(s0, s1);
    }

    // s.w = this CTA's rows of the product, or of b less the product
    __device__ void gather(bool residual) {
        constexpr int kSlices = kThreads / 16;
        // threads: 16 rows x 32 slices at a time
        const int lr = threadIdx.x & 15, sl = threadIdx.x >> 4;
        for (int rb = 0; rb < rows; rb += 16) {
            const int r = rb + lr;
            double t = 0.0;
            if (r < rows)
                for (int q = sl; q < a.splits; q += kSlices)
                    t += __ldcg(a.part + (int64_t)q * a.tiles * kTileRows + r0 + r);
            if (r < rows) s.red[sl][r] = t;
        }
        __syncthreads();
        for (int r = threadIdx.x; r < rows; r += kThreads) {
            double t = 0.0;
            const int ns = min(kSlices, a.splits);
            for (int q = 0; q < ns; ++q) t += s.red[q][r];
            s.w[r] = residual ? s.b[r] - t : t;
        }
        __syncthreads();
    }

    // out[q] = sum over the grid of u . v over the CTAs' rows, one warp per q
    // < cnt; slot: a place of its own in the exchange buffer
    template <typename F>
    __device__ bool dots(int cnt, int slot, F value, double *out) {
        const int lane = threadIdx.x & 31, q = threadIdx.x >> 5;
        if (q < cnt) {
            double t = 0.0;
            for (int r = lane; r < rows; r += 32) t += value(q, r);
            t = warp_sum(t);
            if (lane == 0) a.dots[((int64_t)slot * KM + q) * gridDim.x + blockIdx.x] = t;
        }
        if (!barrier()) return false;
        if (q < cnt) {
            double t = 0.0;
            for (int b = lane; b < (int)gridDim.x; b += 32) t += __ldcg(a.dots + ((int64_t)slot * KM + q) * gridDim.x + b);
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
        product(x, 1.0);
        if (!barrier()) return false;
        gather(true);
        publish(a.w, s.w);
        if (!dots(1, 2, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return false;
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
        __syncthreads();
        // |b| with the first residual's barriers
        product(a.x, 1.0);
        if (!dots(1, 0, [&](int, int r) { return s.b[r] * s.b[r]; }, s.sum)) return leave(kSmallTimeout);
        ++st.matvecs;
        const double bn = sqrt(s.sum[0]);
        if (!isfinite(bn)) return leave(kSmallNaN);
        if (bn == 0.0) {
            for (int r = threadIdx.x; r < rows; r += kThreads) a.x[r0 + r] = 0.0;
            return leave(kSmallOk);
        }
        gather(true);
        publish(a.w, s.w);
        if (!dots(1, 1, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return leave(kSmallTimeout);
        double beta = sqrt(s.sum[0]);
        if (!isfinite(beta)) return leave(kSmallNaN);
        if (beta == 0.0) return leave(kSmallOk);
        bool check_failed = false;  // an estimate within the tolerance whose true residual was not
        for (;;) {
            double norm = beta;  // of the vector in a.w
            if (threadIdx.x <= KM) s.g[threadIdx.x] = threadIdx.x == 0 ? beta : 0.0;
            double bea = 0.0;
            bool stopped = false;  // xcur holds the estimate's solution
            for (int j = 0; j < a.m; ++j) {
                const double inv = 1.0 / norm;
                for (int r = threadIdx.x; r < rows; r += kThreads) s.V[j][r] = s.w[r] * inv;
                product(a.w, inv);
                if (!barrier()) return leave(kSmallTimeout);
                ++st.matvecs;
                gather(false);
                if (!dots(j + 1, 0, [&](int q, int r) { return s.V[q][r] * s.w[r]; }, s.h1)) return leave(kSmallTimeout);
                for (int r = threadIdx.x; r < rows; r += kThreads) {
                    double t = s.w[r];
                    for (int q = 0; q <= j; ++q) t -= s.h1[q] * s.V[q][r];
                    s.w[r] = t;
                }
                __syncthreads();
                if (!dots(j + 1, 1, [&](int q, int r) { return s.V[q][r] * s.w[r]; }, s.h2)) return leave(kSmallTimeout);
                for (int r = threadIdx.x; r < rows; r += kThreads) {
                    double t = s.w[r];
                    for (int q = 0; q <= j; ++q) t -= s.h2[q] * s.V[q][r];
                    s.w[r] = t;
                    a.w[r0 + r] = t;
                }
                __syncthreads();
                if (!dots(1, 2, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return leave(kSmallTimeout);
                norm = sqrt(s.sum[0]);
                if (threadIdx.x == 0) {
                    double *h = s.H[j];
                    bool finite = isfinite(norm);
                    for (int r = 0; r <= j; ++r) {
                        h[r] = s.h1[r] + s.h2[r];
                        finite = finite && isfinite(h[r]);
                    }
                    double hn = norm;
                    for (int r = 0; r < j; ++r) rot(h[r], h[r + 1], s.cs[r], s.sn[r]);
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
                product(a.xcur, 1.0);
                if (!barrier()) return leave(kSmallTimeout);
                ++st.matvecs;
                gather(true);
                if (!dots(1, 0, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return leave(kSmallTimeout);
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
                if (!dots(1, 0, [&](int, int r) { return s.w[r] * s.w[r]; }, s.sum)) return leave(kSmallTimeout);
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
    const int per = (int)((a.n + gridDim.x - 1) / gridDim.x);
    const int r0 = min((int)a.n, (int)blockIdx.x * per), r1 = min((int)a.n, r0 + per);
    Solver v{a, s, r0, r1 - r0};
    v.run();
}

}  // namespace

bool gmres_small_supported(int64_t n, int m, int sm_count) {
    return n >= 1 && m >= 1 && m <= KM && n <= kSmallMaxN && (n + sm_count - 1) / sm_count <= kSmallRows;
}

// The split of the product: about one part per warp of the grid, at least 8 columns each.
static void small_split(int64_t n, int sm_count, int *tiles, int *splits, int *cols) {
    *tiles = (int)((n + kTileRows - 1) / kTileRows);
    int sp = sm_count * kWarps / *tiles;
    sp = std::max(1, std::min<int>(sp, (int)(n / 8)));
    *cols = (int)((n + sp - 1) / sp);
    *splits = (int)((n + *cols - 1) / *cols);
}

int64_t gmres_small_work(int64_t n, int sm_count) {
    int tiles, splits, cols;
    small_split(n, sm_count, &tiles, &splits, &cols);
    return (int64_t)splits * tiles * kTileRows + 3LL * KM * sm_count + 2 * n + 8;
}

cudaError_t launch_gmres_small(SmallGmresArgs a, double *work, int sm_count, cudaStream_t st) {
    small_split(a.n, sm_count, &a.tiles, &a.splits, &a.cols);
    a.part = work;
    a.dots = a.part + (int64_t)a.splits * a.tiles * kTileRows;
    a.w = a.dots + 3LL * KM * sm_count;
    a.xcur = a.w + a.n;
    cudaError_t e = cudaFuncSetAttribute(gmres_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(Shared));
    if (e == cudaSuccess) e = cudaMemsetAsync(a.barrier, 0, sizeof(unsigned), st);
    if (e != cudaSuccess) return e;
    void *args[] = {&a};
    return cudaLaunchCooperativeKernel(reinterpret_cast<void *>(gmres_small_kernel), dim3(sm_count), dim3(kThreads), args,
                                       sizeof(Shared), st);
}

}  // namespace rf
