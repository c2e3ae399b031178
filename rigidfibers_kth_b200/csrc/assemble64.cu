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
// tensor cores, which share it, 9.5 %) with 14 resident warps per SM (124
// registers, 54 KB of shared memory per CTA: four CTAs); the stalls that are
// left are fixed latencies (2.2 warps per issue) and the pipe itself (1.6).
// Unrolling the recursion and P3 over its lanes' items made the code exceed
// the instruction cache (4.6 of 7 warps per issue without an instruction,
// 35.8 ms at M = 4000); with the recursion above n = 8 and P3's rows as
// loops that stall is 0.1.  P3 with one lane per (target, k, l), each loading
// its own neighbours' projections, took 10 % longer (twice the shared-memory
// loads).
#include <algorithm>

#include "rf_kernels.h"

namespace rf {

namespace {

constexpr int kTI = 4;      // targets per warp
constexpr int kWarps = 4;   // warps per CTA

template <int N>
struct Dims64 {
    static constexpr int NL = N + 1;
    static constexpr int NU = N + 1, NV = N + 3;
    static constexpr int NC = NU + NV;              // scalars per point
    static constexpr int COLS = kTI * NC;           // product columns: a multiple of 8
    static constexpr int TILES = COLS / 8;
    static constexpr int KST = 9;                   // stride of a scalar's projections (8 rows)
    static constexpr int PST = NC * KST + (NC * KST % 16 <= 6 ? 6 : 22) - NC * KST % 16;  // of a pair's: 6 mod 16
    static constexpr int TH = kTI * PST;
    static constexpr int RT = kTI * 3 * N;          // staged rows
    static constexpr int CT = 3 * N;                // staged columns
    static constexpr int PAN = 2 * CT * kTI * 3;    // staged panel entries
};

// points of a row of G: a stride of 4 mod 8 keeps the tensor-core operand
// loads and the point-order stores free of bank conflicts
__host__ __device__ constexpr int ldq_of(int LQ) { return ((LQ + 3) / 8) * 8 + 4; }

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

// Coefficients of row k of the factored block: <s f>_k and <s^2 f>_k from
// rows k - 2 .. k + 2 (Bonnet), and v = g1 (AI I + D X^T + p Z^T) +
// t (g1 Y + g2 Q)^T.
struct RowTab {
    double al, be;        // <s f>_k = al f_{k+1} + be f_{k-1}
    double c2p, c20, c2m; // <s^2 f>_k = c2p f_{k+2} + c20 f_k + c2m f_{k-2}
    double g1, g2;
};

struct GStoreUV {
    double *g;   // column 0 of the point's pair, at the point
    int ldq, nu;
    __device__ __forceinline__ void u(int p, double v) const { g[p * ldq] = v; }
    __device__ __forceinline__ void v(int p, double v) const { g[(nu + p) * ldq] = v; }
};

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
    if (tid < NL + 2) {
        const int k = tid < NL ? tid : tid - NL;
        auto al = [](int r) { return (r + 1.0) / (2.0 * r + 1.0); };
        auto be = [](int r) { return r / (2.0 * r + 1.0); };
        RowTab r;
        r.al = al(k);
        r.be = be(k);
        r.c2p = al(k) * al(k + 1);
        r.c20 = al(k) * be(k + 1) + (k > 0 ? be(k) * al(k - 1) : 0.0);
        r.c2m = k > 1 ? be(k) * be(k - 1) : 0.0;
        if (tid < NL) {
            r.g1 = k >= 2 ? tab.gamma[k] : 0.0;
            r.g2 = k >= 2 ? -tab.gamma[k] * tab.Ek[k] : tab.D1;
        } else {
            r.g1 = (k == 0 ? 0.5 : 1.5) / tab.d;
            r.g2 = k == 0 ? 0.0 : -1.5 / tab.d;
        }
        s_row[tid] = r;
    }
    for (int t = tid; t < Far<N>::kCoef; t += kWarps * 32) s_far[t] = Far<N>::coef(t);
    if (tid < NL * 3) {
        const int m = tid / 3, p = m - 2 * (tid % 3);
        s_leg[tid] = p >= 0 ? leg_scale(m) * leg_coef(m, p) : 0.0;
    }
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
        {
            double d[D::TILES][2];
#pragma unroll
            for (int t = 0; t < D::TILES; ++t) d[t][0] = d[t][1] = 0.0;
            const double *bsrc = s_g + (lane >> 2) * LDQ + (lane & 3);
#pragma unroll
            for (int s = 0; s < KSMAX; ++s)
                if (s < KS) {
#pragma unroll
                    for (int t = 0; t < D::TILES; ++t)
                        dmma_8x8x4(d[t][0], d[t][1], afrag[s], bsrc[t * 8 * LDQ + 4 * s], d[t][0], d[t][1]);
                }
            __syncwarp();  // every lane's operands read: the projections take the place of G
#pragma unroll
            for (int t = 0; t < D::TILES; ++t) {
                const int cc = t * 8 + 2 * (lane & 3);  // even: both columns are of one pair
                double *o = s_th + cc / NC * D::PST + cc % NC * KST + (lane >> 2);
                o[0] = d[t][0];
                o[KST] = d[t][1];
            }
        }
        __syncwarp();
        // ---------------- P3: rows k in turn, the projections of rows k - 2 .. k + 2 kept in registers
        if (item3) {
            const double *x = s_tgt + ti3 * 6;
            const double t0 = x[3], t1 = x[4], t2 = x[5];
            const double D0 = x[0] - xs[0], D1 = x[1] - xs[1], D2 = x[2] - xs[2];
            const double dt = D0 * t0 + D1 * t1 + D2 * t2, tt = t0 * t0 + t1 * t1 + t2 * t2,
                         pt = ts[0] * t0 + ts[1] * t1 + ts[2] * t2;
            const double l0 = s_leg[3 * m3], l1 = s_leg[3 * m3 + 1], l2 = s_leg[3 * m3 + 2];
            const double *U = s_th + ti3 * D::PST + m3 * KST, *V = U + NU * KST;
            const int o1 = (max(m3 - 2, 0) - m3) * KST, o2 = (max(m3 - 4, 0) - m3) * KST;
            // Legendre combination m of the scalars at f, f - 2, f - 4
            auto leg = [&](const double *f) { return fma(l2, f[o2], fma(l1, f[o1], l0 * f[0])); };
            double r0m2, r0m1 = 0.0, r0 = 0.0, r0p1 = leg(V), r0p2 = leg(V + 1);         // <cRR>, rows k-2 .. k+2
            double c0m1, c0 = 0.0, c0p1 = leg(V + KST);                                  // -<cPR>, rows k-1 .. k+1
            const bool own = ti3 == self;
            double *dst = s_blk + 3 * (m3 - 1) * D::RT + ti3 * 3 * N;
            double *dpan = s_pan + 3 * (m3 - 1) * (kTI * 3) + ti3 * 3;
            double *acc = s_acc + ti3 * ACCN * 3;
#pragma unroll 1
            for (int k = 0; k <= N; ++k) {
                r0m2 = r0m1; r0m1 = r0; r0 = r0p1; r0p1 = r0p2; r0p2 = leg(V + k + 2);
                c0m1 = c0; c0 = c0p1; c0p1 = leg(V + KST + k + 1);
                if (!PANELS && k == 0) continue;
                const double E = leg(V + 2 * KST + k), AI = leg(U + k);
                const RowTab *rt = s_row + k;
                const double al = rt->al, be = rt->be;
                const double R1 = fma(al, r0p1, be * r0m1);
                const double R2 = fma(rt->c2p, r0p2, fma(rt->c20, r0, rt->c2m * r0m2));
                const double C0 = -c0, C1 = -fma(al, c0p1, be * c0m1);
                const double X0 = fma(r0, D0, fma(R1, t0, C0 * ts[0])), X1 = fma(r0, D1, fma(R1, t1, C0 * ts[1])),
                             X2 = fma(r0, D2, fma(R1, t2, C0 * ts[2]));
                const double Y0 = fma(R1, D0, fma(R2, t0, C1 * ts[0])), Y1 = fma(R1, D1, fma(R2, t1, C1 * ts[1])),
                             Y2 = fma(R1, D2, fma(R2, t2, C1 * ts[2]));
                const double Z0 = fma(C0, D0, fma(C1, t0, E * ts[0])), Z1 = fma(C0, D1, fma(C1, t1, E * ts[1])),
                             Z2 = fma(C0, D2, fma(C1, t2, E * ts[2]));
                // Q = theta t
                const double Q0 = fma(AI, t0, fma(dt, X0, fma(tt, Y0, pt * Z0))),
                             Q1 = fma(AI, t1, fma(dt, X1, fma(tt, Y1, pt * Z1))),
                             Q2 = fma(AI, t2, fma(dt, X2, fma(tt, Y2, pt * Z2)));
                // g1 theta + g2 t Q^T to out (l >= 1), or its product with f added to sum (l = 0)
                auto block = [&](double g1, double g2, double *out, int ldo, double *sum, bool identity) {
                    const double y0 = fma(g1, Y0, g2 * Q0), y1 = fma(g1, Y1, g2 * Q1), y2 = fma(g1, Y2, g2 * Q2);
                    const double gD0 = g1 * D0, gD1 = g1 * D1, gD2 = g1 * D2;
                    const double gp0 = g1 * ts[0], gp1 = g1 * ts[1], gp2 = g1 * ts[2], gA = g1 * AI;
                    double v[9];  // [column][row]
                    v[0] = fma(gD0, X0, fma(t0, y0, fma(gp0, Z0, gA)));
                    v[1] = fma(gD1, X0, fma(t1, y0, gp1 * Z0));
                    v[2] = fma(gD2, X0, fma(t2, y0, gp2 * Z0));
                    v[3] = fma(gD0, X1, fma(t0, y1, gp0 * Z1));
                    v[4] = fma(gD1, X1, fma(t1, y1, fma(gp1, Z1, gA)));
                    v[5] = fma(gD2, X1, fma(t2, y1, gp2 * Z1));
                    v[6] = fma(gD0, X2, fma(t0, y2, gp0 * Z2));
                    v[7] = fma(gD1, X2, fma(t1, y2, gp1 * Z2));
                    v[8] = fma(gD2, X2, fma(t2, y2, fma(gp2, Z2, gA)));
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
                if (k > 0) block(rt->g1, rt->g2, dst + 3 * (k - 1), D::RT, acc + 3 * (k - 1), k == m3);
                if (PANELS && k < 2) {
                    const RowTab *rp = s_row + NL + k;
                    block(rp->g1, rp->g2, dpan + k * D::CT * kTI * 3, kTI * 3, acc + 3 * (N + k), false);
                }
            }
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
