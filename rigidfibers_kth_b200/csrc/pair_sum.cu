// pair_sum.cu - K3 and K7: the sum over all other fibers of the inner integral
// against their force expansion, at every target point, then projected.
//
//   velocities (K3): u_q = sum_j int G(xbar_q - x_j - s t_j) f_j(s) ds with
//     f_j = ExtForce / 2 + sum_l a_j^l P_l, projected onto P_0 and P_1.
//     Reference: fortran/coeffs_and_vels.f90:543-746 (compute_velocities[_an]),
//     Int_analytical.f90:772-850, 905-937, quadrature.f90:166-259;
//     src/kernels/update_velocities.cu:101-191.
//   matrix-free product y = A x (K7, rf_matvec_free): f_j from x alone,
//     projected onto P_1 .. P_N and mapped by the block formula (k = 1: D1 t (t
//     . IF); k >= 2: gamma_k (IF - E_k t (t . IF))).  Reference: mat_prod,
//     fortran/matrix_assembly.f90:159-265.  A is never formed: memory O(M).
//
// Mapping.  A CTA owns some targets (four of the usual 24 points) and a chunk of
// sources, thread (ti, q) one target point; the sources are staged in shared memory in batches, with what
// all points of the GPU share of a source formed once per CTA: the force's
// monomial coefficients F_p (P_l written out) and pb . F_p, or for the numeric
// integral its weighted values at the source's Gauss points.  Then, with u_p
// and v_p of the point (rf_device.cuh; far points by the backward recursion),
//   int G f = sum_p u_p F_p + aR R0 + aP pb,
//   aR = sum_p v_p R0.F_p - v_{p+1} pb.F_p,  aP = sum_p v_{p+2} pb.F_p - v_{p+1} R0.F_p:
// no Legendre combinations of the moments and no tensors per point.  Per-chunk
// partial sums are added in chunk order (deterministic).
//
// What bounds it: the FP64 pipe (69 % busy on an M = 1000 cloud, 14 resident
// warps per SM, the remaining stalls fixed latencies), with 21 of 32 lanes at
// work where near and far points share a warp.  Device times before (each
// thread formed the Legendre combinations of the moments, loaded the
// source's coefficients itself and evaluated the closed forms everywhere) and
// now: velocities at M = 4000 24.8 -> 13.8 ms, M = 1000 1.71 -> 1.13 ms,
// numeric M = 300 0.30 -> 0.14 ms (there the source's force at its points was
// formed by every target point, with a division and a root per point pair).
#include <algorithm>

#include "rf_kernels.h"

namespace rf {

namespace {

// Targets per CTA: at least four, and at fewer than 24 points a fiber as many as
// fill two or three warps, whichever leaves fewer lanes without a point (four
// targets left 20 of 32 at 3 points, 28 of 64 at 9, 16 of 64 at 12).
// Velocities, M = 800, N = 5: 3 points 357 -> 156 us, 9 points 651 -> 370, 12
// points 630 -> 481, 18 points 805 -> 742.
constexpr int kPoints = 96;
constexpr int kMinTI = 4;
constexpr int targets_of(int LQ) {
    const int two = 64 / LQ, three = kPoints / LQ;
    return three <= kMinTI ? kMinTI : two >= kMinTI && 3 * two >= 2 * three ? two : three;
}
static_assert(targets_of(3) == 32 && targets_of(9) == 7 && targets_of(15) == 4 && targets_of(24) == 4, "");
constexpr int kBatch = 16;  // analytic: sources staged at a time
constexpr int kBatchNum = 4;

constexpr int round32(int v) { return (v + 31) / 32 * 32; }

struct PairSumArgs {
    int M, LQ, TI;             // TI: targets per CTA
    int t0, t1;                // target fibers [t0, t1)
    const double *pos, *ori;
    const double *coeffs;      // n: the sources' coefficients
    const Tables *tab;
    double *part;              // [nchunks][stride]
    int64_t stride;
    int chunk;
};

// staged analytic source: centre, direction, F_p, pb . F_p
template <int N>
struct Source {
    double x[3], t[3], F[N + 1][3], h[N + 1];
    double pad[(N + 1) % 2 == 0 ? 0 : 1];
};
template <int N>
struct alignas(16) SourceA : Source<N> {};

// contraction of the scalars with the source's force, as they are formed
template <int N, typename SRC>
struct ForceSum {
    const SRC &s;
    double g[N + 1];  // R0 . F_p
    double U0 = 0.0, U1 = 0.0, U2 = 0.0, aR = 0.0, aP = 0.0;
    __device__ __forceinline__ ForceSum(const SRC &src, const double *R) : s(src) {
#pragma unroll
        for (int p = 0; p <= N; ++p) g[p] = fma(R[0], s.F[p][0], fma(R[1], s.F[p][1], R[2] * s.F[p][2]));
    }
    __device__ __forceinline__ void u(int p, double v) {
        U0 = fma(v, s.F[p][0], U0);
        U1 = fma(v, s.F[p][1], U1);
        U2 = fma(v, s.F[p][2], U2);
    }
    __device__ __forceinline__ void v(int p, double v) {
        if (p <= N) aR = fma(v, g[p <= N ? p : 0], aR);
        if (p >= 1 && p <= N + 1) {
            aR = fma(-v, s.h[p - 1], aR);
            aP = fma(-v, g[p - 1], aP);
        }
        if (p >= 2) aP = fma(v, s.h[p - 2], aP);
    }
};

// MAXT / MINB: threads and resident CTAs per SM the instance is compiled for
template <int N, bool NUMERIC, bool MATFREE, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB) pair_sum_kernel(PairSumArgs a) {
    constexpr int NL = N + 1;
    using Src = SourceA<N>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int LQ = a.LQ, TI = a.TI, nthreads = blockDim.x, tid = threadIdx.x;
    const Tables &tab = *a.tab;
    // analytic: kBatch sources, then the recursion's table; numeric: kBatchNum
    // x LQ x (point, weighted force); at the end: TI x LQ x 3 sums
    Src *s_src = reinterpret_cast<Src *>(smem_raw);
    double *s_far = reinterpret_cast<double *>(s_src + kBatch);
    double *s_num = reinterpret_cast<double *>(smem_raw);
    double *s_u = reinterpret_cast<double *>(smem_raw);
    if (!NUMERIC)
        for (int t = tid; t < Far<N>::kCoef; t += nthreads) s_far[t] = Far<N>::coef(t);
    const int i0 = a.t0 + blockIdx.x * TI;  // first target of the tile (global index)
    const int ti = tid / LQ, q = tid - ti * LQ;
    const int i = i0 + ti;
    const bool live = ti < TI && i < a.t1;
    double xb[3] = {0.0, 0.0, 0.0};
    if (live) {
        const double *xc = a.pos + 3 * i, *tc = a.ori + 3 * i;
        const double sq = tab.pv[q];
#pragma unroll
        for (int c = 0; c < 3; ++c) xb[c] = fadd(xc[c], fmul(sq, tc[c]));
    }
    const double eps2 = tab.eps2;
    double us[3] = {0.0, 0.0, 0.0};
    const int j0 = blockIdx.y * a.chunk, j1 = min(a.M, j0 + a.chunk);
    constexpr int BATCH = NUMERIC ? kBatchNum : kBatch;
    for (int jb = j0; jb < j1; jb += BATCH) {
        const int nj = min(BATCH, j1 - jb);
        __syncthreads();  // the batch before has been read
        if (!NUMERIC) {
            // one thread per (source, axis) for x, t and F, then pb . F
            for (int e = tid; e < nj * 3; e += nthreads) {
                const int r = e / 3, c = e - 3 * r, j = jb + r;
                s_src[r].x[c] = a.pos[3 * j + c];
                s_src[r].t[c] = a.ori[3 * j + c];
                double f[NL];
                f[0] = MATFREE ? 0.0 : tab.half_force[c];
#pragma unroll
                for (int l = 1; l <= N; ++l) f[l] = leg_scale(l) * a.coeffs[((int64_t)j * N + (l - 1)) * 3 + c];
#pragma unroll
                for (int p = 0; p <= N; ++p) {
                    double F = 0.0;
#pragma unroll
                    for (int l = 0; l <= N; ++l)
                        if (l >= p && leg_coef(l, p) != 0) F = fma(leg_coef(l, p), f[l], F);
                    s_src[r].F[p][c] = F;
                }
            }
            __syncthreads();
            for (int e = tid; e < nj * NL; e += nthreads) {
                const int r = e / NL, p = e - NL * r;
                const Src &s = s_src[r];
                s_src[r].h[p] = fma(s.t[0], s.F[p][0], fma(s.t[1], s.F[p][1], s.t[2] * s.F[p][2]));
            }
        } else {
            // the source's Gauss points and the force there times the weight
            for (int e = tid; e < nj * LQ; e += nthreads) {
                const int r = e / LQ, sidx = e - LQ * r, j = jb + r;
                const double sp = tab.pv[sidx], w = tab.wv[sidx];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    double f = MATFREE ? 0.0 : tab.half_force[c];
#pragma unroll
                    for (int l = 1; l <= N; ++l)
                        f = fma(a.coeffs[((int64_t)j * N + (l - 1)) * 3 + c], tab.P[l][sidx], f);
                    s_num[6 * e + c] = fma(a.ori[3 * j + c], sp, a.pos[3 * j + c]);
                    s_num[6 * e + 3 + c] = w * f;
                }
            }
        }
        __syncthreads();
        if (!live) continue;
#pragma unroll 1
        for (int r = 0; r < nj; ++r) {
            if (jb + r == i) continue;
            if (!NUMERIC) {
                const Src &s = s_src[r];
                const double R[3] = {fsub(xb[0], s.x[0]), fsub(xb[1], s.x[1]), fsub(xb[2], s.x[2])};
                const double b = fmul(-2.0, fadd(fadd(fmul(s.t[0], R[0]), fmul(s.t[1], R[1])), fmul(s.t[2], R[2])));
                const double c = fadd(fadd(fmul(R[0], R[0]), fmul(R[1], R[1])), fmul(R[2], R[2]));
                ForceSum<N, Src> f(s, R);
                if (far_point(b, c)) moments_far_fp64<N>(b, c, eps2, s_far, f);
                else moments_near_uv<N>(b, c, eps2, f);
                us[0] += fma(f.aR, R[0], fma(f.aP, s.t[0], f.U0));
                us[1] += fma(f.aR, R[1], fma(f.aP, s.t[1], f.U1));
                us[2] += fma(f.aR, R[2], fma(f.aP, s.t[2], f.U2));
            } else {
                const double *y = s_num + 6 * LQ * r;
                const double e2 = 2.0 * eps2, e6 = 6.0 * eps2;
                // the source's own sum first: 48 additions a source straight into the
                // running sum left rms errors 1.5 times as large (M = 2000)
                double u0 = 0.0, u1 = 0.0, u2 = 0.0;
#pragma unroll 2
                for (int k = 0; k < LQ; ++k, y += 6) {
                    const double Rx = xb[0] - y[0], Ry = xb[1] - y[1], Rz = xb[2] - y[2];
                    const double ir = rsqrt_pos(fma(Rx, Rx, fma(Ry, Ry, Rz * Rz)));
                    const double ir2 = ir * ir, ir3 = ir2 * ir;
                    const double diag = fma(e2, ir3, ir), off = ir3 * fma(-e6, ir2, 1.0);
                    const double rf = fma(Rx, y[3], fma(Ry, y[4], Rz * y[5])) * off;
                    u0 = fma(diag, y[3], fma(Rx, rf, u0));
                    u1 = fma(diag, y[4], fma(Ry, rf, u1));
                    u2 = fma(diag, y[5], fma(Rz, rf, u2));
                }
                us[0] += u0;
                us[1] += u1;
                us[2] += u2;
            }
        }
    }
    __syncthreads();
    if (ti < TI) {
#pragma unroll
        for (int c = 0; c < 3; ++c) s_u[3 * tid + c] = us[c];
    }
    __syncthreads();
    if (!MATFREE) {
        // IF_k = sum_q w_q P_k(s_q) u_q, k = 0, 1
        for (int t = tid; t < TI * 6; t += nthreads) {
            const int gt = t / 6, k = t % 6 / 3, c = t % 3;
            if (i0 + gt >= a.t1) continue;
            double s = 0.0;
            for (int qq = 0; qq < LQ; ++qq) {
                const double w = tab.wv[qq] * (k ? tab.pv[qq] : 1.0);
                s = fma(w, s_u[3 * (gt * LQ + qq) + c], s);
            }
            a.part[(int64_t)blockIdx.y * a.stride + (int64_t)(i0 + gt) * 6 + 3 * k + c] = s;
        }
        return;
    }
    for (int t = tid; t < TI * N; t += nthreads) {
        const int gt = t / N, k = t % N + 1;
        const int it = i0 + gt;
        if (it >= a.t1) continue;
        double IF[3] = {0.0, 0.0, 0.0};
        for (int qq = 0; qq < LQ; ++qq) {
            const double w = tab.wv[qq] * tab.P[k][qq];
            const double *uq = s_u + 3 * (gt * LQ + qq);
#pragma unroll
            for (int c = 0; c < 3; ++c) IF[c] = fma(w, uq[c], IF[c]);
        }
        const double *tc = a.ori + 3 * it;
        const double tIF = tc[0] * IF[0] + tc[1] * IF[1] + tc[2] * IF[2];
        double *dst = a.part + (int64_t)blockIdx.y * a.stride + ((int64_t)it * N + (k - 1)) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            dst[c] = k == 1 ? tab.D1 * tIF * tc[c] : tab.gamma[k] * (IF[c] - tab.Ek[k] * tIF * tc[c]);
    }
}

// y = x + the per-chunk partials, added in chunk order
__global__ void matfree_finish_kernel(int64_t n, int nchunks, const double *part, const double *x, double *y) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= n) return;
    double s = x[r];
    for (int c = 0; c < nchunks; ++c) s += part[(int64_t)c * n + r];
    y[r] = s;
}

// resident CTAs per SM of the usual sizes (up to 24 points)
constexpr int kMinB = 5;

template <int N, bool NUMERIC, bool MATFREE>
cudaError_t launch_n(const PairSumArgs &a, int nchunks, cudaStream_t st) {
    const int threads = round32(a.TI * a.LQ);
    const size_t src = NUMERIC ? sizeof(double) * 6 * kBatchNum * a.LQ
                               : sizeof(SourceA<N>) * kBatch + sizeof(double) * Far<N>::kCoef;
    const size_t smem = std::max(src, sizeof(double) * 3 * a.TI * (size_t)a.LQ);
    auto kern = threads <= kPoints ? pair_sum_kernel<N, NUMERIC, MATFREE, kPoints, kMinB>
                                   : pair_sum_kernel<N, NUMERIC, MATFREE, kMinTI * kMaxLQ, 2>;
    kern<<<dim3((a.t1 - a.t0 + a.TI - 1) / a.TI, nchunks), threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <bool MATFREE>
cudaError_t launch_pair_sum(const PairSumArgs &a, int N, bool numeric, int nchunks, cudaStream_t st) {
    switch (N) {
#define RF_CASE(n) \
    case n: return numeric ? launch_n<n, true, MATFREE>(a, nchunks, st) : launch_n<n, false, MATFREE>(a, nchunks, st);
        RF_CASE(1) RF_CASE(2) RF_CASE(3) RF_CASE(4) RF_CASE(5) RF_CASE(6) RF_CASE(7) RF_CASE(8)
#undef RF_CASE
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

int pair_sum_chunks(int M, int LQ, int sm_count) {
    const int TI = targets_of(LQ);
    return pick_chunks(M, (M + TI - 1) / TI, kMinB * (int64_t)sm_count, 1);
}

cudaError_t launch_velocity(const VelArgs &a, bool numeric, int nchunks, cudaStream_t st) {
    return launch_pair_sum<false>({a.M, a.LQ, targets_of(a.LQ), a.t0, a.t1, a.pos, a.ori, a.coeffs, a.tab, a.part, 6LL * a.M, a.chunk},
                                  a.N, numeric, nchunks, st);
}

cudaError_t launch_matfree(const MatfreeArgs &a, bool numeric, int nchunks, const double *x, double *y,
                           cudaStream_t st) {
    cudaError_t e = launch_pair_sum<true>({a.M, a.LQ, targets_of(a.LQ), 0, a.M, a.pos, a.ori, a.x, a.tab, a.part, a.n, a.chunk}, a.N,
                                          numeric, nchunks, st);
    if (e != cudaSuccess) return e;
    matfree_finish_kernel<<<(unsigned)((a.n + 255) / 256), 256, 0, st>>>(a.n, nchunks, a.part, x, y);
    return cudaGetLastError();
}

}  // namespace rf
