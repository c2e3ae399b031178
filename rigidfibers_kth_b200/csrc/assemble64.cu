// assemble64.cu - K1 for the FP64 analytic method, N <= 5: the dense system
// assembled by autonomous warps.
//
// Reference: fortran/matrix_assembly.f90:407-629 (matrix, analytic) and
// 796-905 (right-hand side); Int_analytical.f90:72-288 (inner integral).
//
// A warp owns four target fibers and walks a chunk of sources; the warps of a
// CTA share only the tables, so there is no barrier in the source loop.  Per
// source:
//   P1  lanes = the 4 LQ target points, 32 at a time: the scalars u_p, v_p of
//       the inner integral (rf_device.cuh) into shared memory.  Far points
//       take the backward recursion; the others are listed and then
//       integrated together with the reference's formulas, so that a warp
//       with one near pair does not run both paths in every round;
//   P2  their projections onto P_0 .. P_{N+2} on the FP64 tensor cores
//       (mma.sync m8n8k4): 8 rows x (4 pairs x (2N + 4) scalars);
//   P3  lane = (target, l), l = 0..N, over the rows k: the 3 x 3 blocks from
//       the projections, the pair tensors factored as theta = AI I + D X^T +
//       t Y^T + p Z^T (header of assemble_split.cu), the projections of s f
//       and s^2 f from Bonnet's recursion; the l = 0 lanes sum theta f, f =
//       ExtForce / 2, over the sources (right-hand side, velocity terms);
//   P4  15-column x 60-row blocks (N = 5) written with 16-byte stores.
// The tile kernel (assemble.cu), which this one replaces here, formed the 36
// tensor components at every point (projecting 36 columns per pair, not 14)
// and evaluated the closed forms at every point; it stays for the numeric
// integral, for N > 5 (more than eight projection rows) and for the mixed
// modes that ask for FP64 integrals.  Device time of one assembly with the
// tile kernel and with this one: M = 4000 cloud 50.0 -> 20.9 ms, M = 1000
// cloud 3.36 -> 1.6 ms (30 % of its points take the reference's formulas),
// M = 1000 with N = 2 2.0 -> 1.2 ms, M = 1000 with panels 3.8 -> 2.0 ms.
//
// What bounds it: the FP64 pipe (M = 1000 cloud: 54 % busy and the FP64
// tensor cores, which share it, 9.5 %) with 14 resident warps per SM (122
// registers, 54 KB of shared memory per CTA: four CTAs); the stalls that are
// left are fixed latencies (2.2 warps per issue) and the pipe itself (1.6).
// Unrolling the recursion and P3 over its lanes' items made the code exceed
// the instruction cache (4.6 of 7 warps per issue without an instruction,
// 35.8 ms at M = 4000); with the recursion above n = 8 and P3's rows as
// loops that stall is 0.1.  P3 with one lane per (target, k, l), each loading
// its own neighbours' projections, took 10 % longer (twice the shared-memory
// loads).
#include <algorithm>

#include "pair_block64.cuh"
#include "rf_kernels.h"

namespace rf {

namespace {

constexpr int kWarps = 4;   // warps per CTA

// shared memory of a warp, in doubles: G, or the projections, the staged block
// and the staged panels; then the targets, the right-hand-side sums and the
// list of points for the reference's formulas
template <int N, bool PANELS>
__host__ __device__ constexpr int region_doubles(int LQ) {
    using D = Dims64<N>;
    const int g = D::COLS * ldq_of(LQ);
    const int p3 = (D::TH + 1) / 2 * 2 + D::CT * D::RT + (PANELS ? D::PAN : 0);
    return ((g > p3 ? g : p3) + 1) / 2 * 2;
}
template <int N, bool PANELS>
__host__ __device__ constexpr int warp_doubles(int LQ) {
    return region_doubles<N, PANELS>(LQ) + kTI * 6 + kTI * (N + (PANELS ? 2 : 0)) * 3 + kTI * kMaxLQ / 8;
}

// LQC: the points per fiber when known at compile time (24, the usual 8 x 3), else 0
template <int N, bool PANELS, int KSMAX, int LQC>
__global__ void __launch_bounds__(kWarps * 32, 4) assemble64_kernel(AsmArgs a) {
    using D = Dims64<N>;
    constexpr int NL = D::NL, NC = D::NC, NU = D::NU, KST = D::KST;
    constexpr int ACCN = N + (PANELS ? 2 : 0);  // rows of the l = 0 sums
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int LQ = LQC ? LQC : a.LQ, LDQ = ldq_of(LQ), KS = (LQ + 3) / 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const Tables &tab = *a.tab;

    double *s_pv = reinterpret_cast<double *>(smem_raw);               // kMaxLQ
    RowTab *s_row = reinterpret_cast<RowTab *>(s_pv + kMaxLQ);          // NL block rows, then 2 panel rows
    double *s_leg = reinterpret_cast<double *>(s_row + NL + 2);         // NL x 3: coefficients of p = m, m-2, m-4
    double *s_far = s_leg + NL * 3;                                     // Far<N>::kCoef
    double *s_warp = s_far + Far<N>::kCoef;
    s_warp += (s_warp - s_pv) & 1;                                     // 16-byte aligned
    double *s_wP = s_warp;                                              // 8 x kMaxLQ, until the operands are loaded
    double *s_g = s_warp + warp * warp_doubles<N, PANELS>(LQ);
    double *s_th = s_g;                                                 // after P2: the projections
    double *s_blk = s_th + (D::TH + 1) / 2 * 2;                         // CT x RT
    double *s_pan = s_blk + D::CT * D::RT;                              // 2 x CT x 12
    double *s_tgt = s_g + region_doubles<N, PANELS>(LQ);                // 4 x (x, t)
    double *s_acc = s_tgt + kTI * 6;                                    // 4 x ACCN x 3: N rows of b, 2 of the velocities
    unsigned char *s_list = reinterpret_cast<unsigned char *>(s_acc + kTI * ACCN * 3);

    for (int t = tid; t < kMaxLQ; t += kWarps * 32) s_pv[t] = t < LQ ? tab.pv[t] : 0.0;
    for (int t = tid; t < 8 * kMaxLQ; t += kWarps * 32) {
        const int m = t / kMaxLQ, q = t % kMaxLQ;
        s_wP[t] = (m <= N + 2 && q < LQ) ? tab.wv[q] * tab.P[m][q] : 0.0;
    }
    block_tables<N>(tab, s_row, s_leg, tid);
    for (int t = tid; t < Far<N>::kCoef; t += kWarps * 32) s_far[t] = Far<N>::coef(t);
    __syncthreads();
    // tensor-core A operands: lane holds w_q P_row(q), row = lane / 4, q = 4 s + lane % 4
    double afrag[KSMAX];
#pragma unroll
    for (int s = 0; s < KSMAX; ++s) afrag[s] = s < KS ? s_wP[(lane >> 2) * kMaxLQ + 4 * s + (lane & 3)] : 0.0;
    __syncthreads();
    const int i0 = a.t0 + (blockIdx.x * kWarps + warp) * kTI;  // first target of the warp (global index)
    if (lane < kTI * 6) {
        const int ti = lane / 6, c = lane % 6, i = i0 + ti;
        s_tgt[lane] = i < a.t1 ? (c < 3 ? a.pos[3 * i + c] : a.ori[3 * i + c - 3]) : (c < 3 ? 0.0 : 1.0);
    }
    if (i0 >= a.t1) return;  // whole warp; no CTA barrier below

    const double eps2 = tab.eps2;
    const int j0 = blockIdx.y * a.chunk, j1 = min(a.M, j0 + a.chunk);
    const int64_t row0 = (int64_t)(i0 - a.t0) * 3 * N;
    const int ntgt = min(kTI, a.t1 - i0);
    const int rows_valid = ntgt * 3 * N;
    const int npts = kTI * LQ;
    for (int e = lane; e < kTI * ACCN * 3; e += 32) s_acc[e] = 0.0;
    // P3: lane = (target, l)
    const int ti3 = lane / NL, m3 = lane - ti3 * NL;
    const bool item3 = lane < kTI * NL;
    __syncwarp();

    // geometry of point `item` for source j: R0, b, c as the reference forms them (not fused)
    auto point = [&](int item, const double *xs, const double *ts, double &b, double &c) {
        const int ti = item / LQ, q = item - ti * LQ;
        const double sq = s_pv[q];
        const double *x = s_tgt + ti * 6;
        const double rx = fsub(fadd(x[0], fmul(sq, x[3])), xs[0]);
        const double ry = fsub(fadd(x[1], fmul(sq, x[4])), xs[1]);
        const double rz = fsub(fadd(x[2], fmul(sq, x[5])), xs[2]);
        b = fmul(-2.0, fadd(fadd(fmul(ts[0], rx), fmul(ts[1], ry)), fmul(ts[2], rz)));
        c = fadd(fadd(fmul(rx, rx), fmul(ry, ry)), fmul(rz, rz));
    };

    for (int j = j0; j < j1; ++j) {
        const double xs[3] = {__ldg(a.pos + 3 * j), __ldg(a.pos + 3 * j + 1), __ldg(a.pos + 3 * j + 2)};
        const double ts[3] = {__ldg(a.ori + 3 * j), __ldg(a.ori + 3 * j + 1), __ldg(a.ori + 3 * j + 2)};
        const int self = j - i0;  // the target that is the source, if in 0..3
        // ---------------- P1
        int nnear = 0;
#pragma unroll 1
        for (int base = 0; base < npts; base += 32) {
            const int item = base + lane;
            const int ti = item / LQ, q = item - ti * LQ;
            const bool in = item < npts;
            const bool live = in && ti < ntgt && ti != self;
            double b = 0.0, c = 1.0;
            if (live) point(item, xs, ts, b, c);
            const bool far = live && far_point(b, c);
            const GStoreUV out{s_g + ti * NC * LDQ + q, LDQ, NU};
            if (far) {
                moments_far_fp64<N>(b, c, eps2, s_far, out);
            } else if (in && !live) {
#pragma unroll
                for (int p = 0; p < NC; ++p) out.g[p * LDQ] = 0.0;
            }
            const bool near = live && !far;
            const unsigned mask = __ballot_sync(0xffffffffu, near);
            if (near) s_list[nnear + __popc(mask & ((1u << lane) - 1u))] = (unsigned char)item;
            nnear += __popc(mask);
        }
        // the points between LQ and the next multiple of 4 are zero for the tensor-core k-steps
        for (int t = lane; t < D::COLS * (4 * KS - LQ); t += 32) {
            const int pad = 4 * KS - LQ;
            s_g[(t / pad) * LDQ + LQ + t % pad] = 0.0;
        }
        __syncwarp();
#pragma unroll 1
        for (int u = lane; u < nnear; u += 32) {
            const int item = s_list[u];
            const int ti = item / LQ, q = item - ti * LQ;
            double b, c;
            point(item, xs, ts, b, c);
            moments_near_uv<N>(b, c, eps2, GStoreUV{s_g + ti * NC * LDQ + q, LDQ, NU});
        }
        __syncwarp();
        // ---------------- P2
        project_pairs<N, KSMAX>(s_g, s_th, afrag, LDQ, KS, lane);
        // ---------------- P3
        if (item3) {
            const bool own = ti3 == self;
            double *dst = s_blk + 3 * (m3 - 1) * D::RT + ti3 * 3 * N;
            double *dpan = s_pan + 3 * (m3 - 1) * (kTI * 3) + ti3 * 3;
            double *acc = s_acc + ti3 * ACCN * 3;
            block_rows<N, PANELS>(s_row, s_leg, s_th + ti3 * D::PST + m3 * KST, m3, s_tgt + ti3 * 6, xs, ts,
                                  [&](int k, const BlockRow &r) {
                // the block to out (l >= 1), or its product with f added to sum (l = 0)
                auto block = [&](double g1, double g2, double *out, int ldo, double *sum, bool identity) {
                    double v[9];
                    r.entries(g1, g2, v);
                    if (own) {  // the fiber itself: the identity in A, nothing else
#pragma unroll
                        for (int e = 0; e < 9; ++e) v[e] = e % 4 == 0 && identity ? 1.0 : 0.0;
                    }
                    if (m3 > 0) {
#pragma unroll
                        for (int e = 0; e < 9; ++e) out[(e / 3) * ldo + e % 3] = v[e];
                    } else if (!own) {
                        const double f0 = tab.half_force[0], f1 = tab.half_force[1], f2 = tab.half_force[2];
#pragma unroll
                        for (int e = 0; e < 3; ++e) sum[e] += fma(v[e], f0, fma(v[3 + e], f1, v[6 + e] * f2));
                    }
                };
                if (k > 0) block(s_row[k].g1, s_row[k].g2, dst + 3 * (k - 1), D::RT, acc + 3 * (k - 1), k == m3);
                if (PANELS && k < 2)
                    block(s_row[NL + k].g1, s_row[NL + k].g2, dpan + k * D::CT * kTI * 3, kTI * 3, acc + 3 * (N + k),
                          false);
            });
        }
        __syncwarp();
        // ---------------- P4: two consecutive rows per lane
        double *Ac = a.A64 + (int64_t)j * D::CT * a.lda + row0;
        if (rows_valid == D::RT) {
#pragma unroll 4
            for (int e = lane; e < D::CT * D::RT / 2; e += 32) {
                const int cl = e / (D::RT / 2), rl = 2 * (e - cl * (D::RT / 2));
                *reinterpret_cast<double2 *>(Ac + (int64_t)cl * a.lda + rl) =
                    *reinterpret_cast<const double2 *>(s_blk + 2 * e);
            }
        } else {
            for (int e = lane; e < D::CT * D::RT; e += 32) {
                const int cl = e / D::RT, rl = e - cl * D::RT;
                if (rl < rows_valid) Ac[(int64_t)cl * a.lda + rl] = s_blk[e];
            }
        }
        if (PANELS) {
            const int64_t prow0 = (int64_t)i0 * 3, col0 = (int64_t)j * D::CT;
            for (int e = lane; e < D::PAN; e += 32) {
                const int w = e / (D::CT * kTI * 3), g = e - w * (D::CT * kTI * 3);
                const int cl = g / (kTI * 3), rl = g - cl * (kTI * 3);
                if (rl < 3 * ntgt) (w ? a.PW64 : a.PV64)[(col0 + cl) * a.ldp + prow0 + rl] = s_pan[e];
            }
        }
        __syncwarp();  // the next source's G takes the place of the staged block
    }
    // per-chunk partial sums: right-hand side [chunk][n] and the l = 0 velocity
    // terms [chunk][6M] (matrix_assembly.f90:874-899)
    for (int e = lane; e < ntgt * ACCN * 3; e += 32) {
        const int ti = e / (ACCN * 3), r = e - ti * ACCN * 3, ii = i0 + ti;
        if (r < 3 * N)
            a.bpart[(int64_t)blockIdx.y * a.n + (int64_t)(ii - a.t0) * 3 * N + r] = -s_acc[e];
        else if (PANELS && a.vpart)
            a.vpart[(int64_t)blockIdx.y * 6 * a.M + (int64_t)ii * 6 + (r - 3 * N)] = s_acc[e];
    }
}

template <int N, bool PANELS, int KSMAX, int LQC>
cudaError_t launch_n(const AsmArgs &a, int nchunks, cudaStream_t st) {
    const size_t smem = sizeof(double) * (kMaxLQ + 3 * (N + 1) + Far<N>::kCoef + 1 +
                                          kWarps * (size_t)warp_doubles<N, PANELS>(a.LQ)) +
                        sizeof(RowTab) * (N + 3);
    auto kern = assemble64_kernel<N, PANELS, KSMAX, LQC>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    const int per = kWarps * kTI;
    kern<<<dim3((a.t1 - a.t0 + per - 1) / per, nchunks), kWarps * 32, smem, st>>>(a);
    return cudaGetLastError();
}

template <int N>
cudaError_t launch_ks(const AsmArgs &a, int nchunks, cudaStream_t st) {
    if (a.LQ == 24) return a.PV64 ? launch_n<N, true, 6, 24>(a, nchunks, st) : launch_n<N, false, 6, 24>(a, nchunks, st);
    if (a.LQ < 24) return a.PV64 ? launch_n<N, true, 6, 0>(a, nchunks, st) : launch_n<N, false, 6, 0>(a, nchunks, st);
    return a.PV64 ? launch_n<N, true, 12, 0>(a, nchunks, st) : launch_n<N, false, 12, 0>(a, nchunks, st);
}

}  // namespace

bool assemble64_supported(int N) { return N >= 1 && N <= 5; }

int assemble64_chunks(int M, int sm_count) {
    return pick_chunks(M, (M + kWarps * kTI - 1) / (kWarps * kTI), 4 * (int64_t)sm_count, 1);
}

cudaError_t launch_assemble64(const AsmArgs &a, int nchunks, cudaStream_t st) {
    switch (a.N) {
        case 1: return launch_ks<1>(a, nchunks, st);
        case 2: return launch_ks<2>(a, nchunks, st);
        case 3: return launch_ks<3>(a, nchunks, st);
        case 4: return launch_ks<4>(a, nchunks, st);
        case 5: return launch_ks<5>(a, nchunks, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace rf
