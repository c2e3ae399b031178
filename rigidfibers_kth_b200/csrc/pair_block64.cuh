// pair_block64.cuh - the FP64 pieces that the plain assembly (assemble64.cu) and
// the near pairs of the split assembly (assemble_split.cu) share: a warp
// integrates four fiber pairs at a time, their points' scalars u_p, v_p
// (rf_device.cuh) staged as G[pair, scalar][point], projected onto P_0 ..
// P_{N+2} on the FP64 tensor cores, and the 3 x 3 blocks formed from the
// projections row by row, lane = (pair, l).
#pragma once

#include "rf_device.cuh"

namespace rf {

constexpr int kTI = 4;      // pairs of a warp

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

// Row tables: rows 0..N of the block, then the two rows of the velocity panels;
// Legendre coefficients sc_m a_mp for p = m, m - 2, m - 4.
template <int N>
__device__ __forceinline__ void block_tables(const Tables &tab, RowTab *s_row, double *s_leg, int tid) {
    constexpr int NL = N + 1;
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
    if (tid < NL * 3) {
        const int m = tid / 3, p = m - 2 * (tid % 3);
        s_leg[tid] = p >= 0 ? leg_scale(m) * leg_coef(m, p) : 0.0;
    }
}

// The projections of a warp's four pairs: G (after a __syncwarp; points from LQ
// to the next multiple of 4 zero) -> th, which may take G's place.
template <int N, int KSMAX>
__device__ __forceinline__ void project_pairs(const double *s_g, double *s_th, const double (&afrag)[KSMAX], int LDQ,
                                              int KS, int lane) {
    using D = Dims64<N>;
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
    __syncwarp();  // every lane's operands read: the projections may take the place of G
#pragma unroll
    for (int t = 0; t < D::TILES; ++t) {
        const int cc = t * 8 + 2 * (lane & 3);  // even: both columns are of one pair
        double *o = s_th + cc / D::NC * D::PST + cc % D::NC * D::KST + (lane >> 2);
        o[0] = d[t][0];
        o[D::KST] = d[t][1];
    }
    __syncwarp();
}

// One row k of a pair's blocks for source weight m: theta = AI I + D X^T + t Y^T
// + p Z^T, Q = theta t.
struct BlockRow {
    double D0, D1, D2, t0, t1, t2, p0, p1, p2;
    double AI, X0, X1, X2, Y0, Y1, Y2, Z0, Z1, Z2, Q0, Q1, Q2;
    // v = g1 theta + g2 t Q^T, [column][row]
    __device__ __forceinline__ void entries(double g1, double g2, double (&v)[9]) const {
        const double y0 = fma(g1, Y0, g2 * Q0), y1 = fma(g1, Y1, g2 * Q1), y2 = fma(g1, Y2, g2 * Q2);
        const double gD0 = g1 * D0, gD1 = g1 * D1, gD2 = g1 * D2;
        const double gp0 = g1 * p0, gp1 = g1 * p1, gp2 = g1 * p2, gA = g1 * AI;
        v[0] = fma(gD0, X0, fma(t0, y0, fma(gp0, Z0, gA)));
        v[1] = fma(gD1, X0, fma(t1, y0, gp1 * Z0));
        v[2] = fma(gD2, X0, fma(t2, y0, gp2 * Z0));
        v[3] = fma(gD0, X1, fma(t0, y1, gp0 * Z1));
        v[4] = fma(gD1, X1, fma(t1, y1, fma(gp1, Z1, gA)));
        v[5] = fma(gD2, X1, fma(t2, y1, gp2 * Z1));
        v[6] = fma(gD0, X2, fma(t0, y2, gp0 * Z2));
        v[7] = fma(gD1, X2, fma(t1, y2, gp1 * Z2));
        v[8] = fma(gD2, X2, fma(t2, y2, fma(gp2, Z2, gA)));
    }
};

// Rows k = 0 .. N (FROM0) or 1 .. N in turn, the projections of rows k - 2 .. k +
// 2 kept in registers; out(k, row).  x: target centre and direction, xs and ts
// the source's; U: the pair's projections at scalar m.
template <int N, bool FROM0, typename OUT>
__device__ __forceinline__ void block_rows(const RowTab *s_row, const double *s_leg, const double *U, int m,
                                           const double *x, const double *xs, const double *ts, OUT &&out) {
    constexpr int KST = Dims64<N>::KST;
    BlockRow r;
    r.t0 = x[3], r.t1 = x[4], r.t2 = x[5];
    r.D0 = x[0] - xs[0], r.D1 = x[1] - xs[1], r.D2 = x[2] - xs[2];
    r.p0 = ts[0], r.p1 = ts[1], r.p2 = ts[2];
    const double dt = r.D0 * r.t0 + r.D1 * r.t1 + r.D2 * r.t2, tt = r.t0 * r.t0 + r.t1 * r.t1 + r.t2 * r.t2,
                 pt = r.p0 * r.t0 + r.p1 * r.t1 + r.p2 * r.t2;
    const double l0 = s_leg[3 * m], l1 = s_leg[3 * m + 1], l2 = s_leg[3 * m + 2];
    const double *V = U + Dims64<N>::NU * KST;
    const int o1 = (max(m - 2, 0) - m) * KST, o2 = (max(m - 4, 0) - m) * KST;
    // Legendre combination m of the scalars at f, f - 2, f - 4
    auto leg = [&](const double *f) { return fma(l2, f[o2], fma(l1, f[o1], l0 * f[0])); };
    double r0m2, r0m1 = 0.0, r0 = 0.0, r0p1 = leg(V), r0p2 = leg(V + 1);  // <cRR>, rows k-2 .. k+2
    double c0m1, c0 = 0.0, c0p1 = leg(V + KST);                           // -<cPR>, rows k-1 .. k+1
#pragma unroll 1
    for (int k = 0; k <= N; ++k) {
        r0m2 = r0m1; r0m1 = r0; r0 = r0p1; r0p1 = r0p2; r0p2 = leg(V + k + 2);
        c0m1 = c0; c0 = c0p1; c0p1 = leg(V + KST + k + 1);
        if (!FROM0 && k == 0) continue;
        const double E = leg(V + 2 * KST + k);
        r.AI = leg(U + k);
        const RowTab *rt = s_row + k;
        const double R1 = fma(rt->al, r0p1, rt->be * r0m1);
        const double R2 = fma(rt->c2p, r0p2, fma(rt->c20, r0, rt->c2m * r0m2));
        const double C0 = -c0, C1 = -fma(rt->al, c0p1, rt->be * c0m1);
        r.X0 = fma(r0, r.D0, fma(R1, r.t0, C0 * r.p0));
        r.X1 = fma(r0, r.D1, fma(R1, r.t1, C0 * r.p1));
        r.X2 = fma(r0, r.D2, fma(R1, r.t2, C0 * r.p2));
        r.Y0 = fma(R1, r.D0, fma(R2, r.t0, C1 * r.p0));
        r.Y1 = fma(R1, r.D1, fma(R2, r.t1, C1 * r.p1));
        r.Y2 = fma(R1, r.D2, fma(R2, r.t2, C1 * r.p2));
        r.Z0 = fma(C0, r.D0, fma(C1, r.t0, E * r.p0));
        r.Z1 = fma(C0, r.D1, fma(C1, r.t1, E * r.p1));
        r.Z2 = fma(C0, r.D2, fma(C1, r.t2, E * r.p2));
        r.Q0 = fma(r.AI, r.t0, fma(dt, r.X0, fma(tt, r.Y0, pt * r.Z0)));
        r.Q1 = fma(r.AI, r.t1, fma(dt, r.X1, fma(tt, r.Y1, pt * r.Z1)));
        r.Q2 = fma(r.AI, r.t2, fma(dt, r.X2, fma(tt, r.Y2, pt * r.Z2)));
        out(k, r);
    }
}

}  // namespace rf
