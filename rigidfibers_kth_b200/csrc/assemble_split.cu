// assemble_split.cu - mixed-precision assembly split by pair distance.
//
// Reference: fortran/matrix_assembly.f90:407-629 (matrix, analytic) and
// 796-905 (right-hand side); Int_analytical.f90:72-288 (inner integral).
//
// The mixed path stores A in FP32: as FP32 words (FP32 paths) or as the two
// 16-bit planes of split storage (BF16 path; the high plane is the BF16
// matrix of the inner solves).  A fiber pair (i, j) is "near"
// when one of target i's quadrature points lies within sqrt(near_c) of source
// j's centre (default c < 6: closer, the FP32 backward recursion loses digits;
// the reference itself switches to forward recursion below 10).  Near pairs
// are integrated in FP64, far pairs in FP32, every moment of a far pair by the
// backward recursion run down to n = 0 (moments_backward_fp32: none of the
// reference's n = 0, 1 closed forms, which cancel for distant pairs and close
// to the source axis).  Three kernels:
//   classify_kernel   one warp per target: near-pair bitmap and per-target
//                     lists in ascending source order;
//   far_pairs_kernel  FP32, lane = target fiber, warp-uniform source, eight
//                     warps per CTA stepping through the sources together:
//                     every lane integrates its own pair over the target's
//                     Gauss points with the projection accumulated in
//                     registers, then stages the 3N x 3N block (split into
//                     its two 16-bit planes where stored so) and the
//                     velocity-panel rows in shared memory, and one lane
//                     hands whole column segments to the copy engine;
//   near_pairs_kernel FP64, a warp per four near pairs of a target, their
//                     points integrated together, the projection on the FP64
//                     tensor cores (mma.sync m8n8k4), as in assemble64.cu.
// A finish kernel sums the per-chunk right-hand-side partials in a fixed order.
//
// Projection without forming the tensors.  The reference forms, per target
// point q and source weight m, G_m(q) = cI I + cRR R0R0 + cPR (pR0 + R0p)
// + cPP pp and projects theta^k_m = sum_q w_q P_k(s_q) G_m(q).  Here
//   cI  = sc_m sum_p a_mp u_p,        u_p = I_p + 2 eps^2 J_p
//   cRR = sc_m sum_p a_mp v_p,        v_p = J_p - 6 eps^2 S_p
//   cPR = -sc_m sum_p a_mp v_{p+1},   cPP = sc_m sum_p a_mp v_{p+2}
// (a_mp, sc_m the Legendre coefficients of Int_analytical.f90:213-288), and
// R0 = D + s_q t with D = x_i - x_j, t = t_i, so every entry of theta is a
// combination of the scalar projections <u_p>_k, <v_p>_k, <s v_p>_k and
// <s^2 v_p>_k times the seven pair tensors I, DD, Dt+tD, tt, pD+Dp, pt+tp,
// pp.  Bonnet's recursion s P_k = ((k+1) P_{k+1} + k P_{k-1}) / (2k+1) holds
// at every point, so <s f>_k = alpha_k <f>_{k+1} + beta_k <f>_{k-1}: the
// per-point work is 2N+4 scalars projected onto P_0..P_{N+2}, the same sums in
// another order.
#include <algorithm>

#include "pair_block64.cuh"
#include "rf_kernels.h"

namespace rf {

namespace {

template <int N>
struct SplitDims {
    static constexpr int NL = N + 1;          // u_p and Legendre indices 0..N
    static constexpr int NV = N + 3;          // v_p, p = 0..N+2
    static constexpr int KW = N + 3;          // projection rows k = 0..N+2
    static constexpr int KWP = KW + (KW & 1); // KW rounded up to even: the weight table's row stride
    static constexpr int NC = NL + NV;        // scalars per Gauss point
    static constexpr int RB = 3 * N;          // rows (and columns) of a pair block
    static constexpr int NRHS = 3 * NL;       // theta^k_0 f, k = 0..N
};

// number of projection rows kept for v_p
__host__ __device__ constexpr int vrows(int N, int p) { return p <= N ? N + 3 : (p == N + 1 ? N + 2 : N + 1); }

__host__ __device__ constexpr double bonnet_a(int k) { return (k + 1.0) / (2.0 * k + 1.0); }
__host__ __device__ constexpr double bonnet_b(int k) { return k / (2.0 * k + 1.0); }

// FP64 moments for the near pairs of the mixed path: the reference formulas
// (Int_analytical.f90:96-207) with ordinary (contracted) arithmetic and the
// loop-constant divisions folded into reciprocals.
template <int N>
__device__ __forceinline__ void moments_near(double b, double c, double *I, double *J, double *S) {
    constexpr int K = N + 3;
    const double xe = 1.0 + b + c, xb = 1.0 - b + c;
    const double iue = rsqrt(xe), iub = rsqrt(xb);
    const double ue = xe * iue, ub = xb * iub;
    const double te = 1.0 + 0.5 * b;
    const double tb = -1.0 + 0.5 * b;
    const double d = c - 0.25 * b * b;
    I[0] = log(fabs((2.0 + b + 2.0 * ue) / (-2.0 + b + 2.0 * ub)));
    I[1] = ue - ub - 0.5 * b * I[0];
    if (d < 1e-14) {
        const double e1 = 1.0 + 0.5 * b, e2 = -1.0 + 0.5 * b;
        J[0] = -0.5 / (e1 * e1) + 0.5 / (e2 * e2);
        J[1] = -iue + iub - 0.5 * b * J[0];
        const double p = 2.0 + b, m = -2.0 + b;
        const double p2 = p * p, m2 = m * m;
        S[0] = -4.0 / (p2 * p2) + 4.0 / (m2 * m2);
        S[1] = -8.0 / (3.0 * p2 * p) + 8.0 / (3.0 * m2 * m) - 0.5 * b * S[0];
    } else {
        const double id = 1.0 / d;
        J[0] = (te * iue - tb * iub) * id;
        J[1] = -iue + iub - 0.5 * b * J[0];
        const double iue3 = iue * iue * iue, iub3 = iub * iub * iub;
        const double id6 = id * (1.0 / 6.0);
        S[0] = ((2.0 + b) * iue3 - (-2.0 + b) * iub3) * id6 + (2.0 / 3.0) * id * J[0];
        S[1] = (-(b + 2.0 * c) * iue3 + (-b + 2.0 * c) * iub3) * id6 - (1.0 / 3.0) * b * id * J[0];
    }
    if (c < 10.0) {
#pragma unroll
        for (int n = 2; n < K; ++n) {
            const double nn = n + 1.0;
            const double r = 1.0 / (1.0 - nn);
            const double sbp = (n % 2 == 1) ? 1.0 : -1.0;
            I[n] = (sbp * r) * ub - r * ue - ((0.5 - (nn - 1.0)) * r) * b * I[n - 1] + ((nn - 2.0) * r) * c * I[n - 2];
            J[n] = I[n - 2] - b * J[n - 1] - c * J[n - 2];
            S[n] = J[n - 2] - b * S[n - 1] - c * S[n - 2];
        }
    } else {
        const double ic = 1.0 / c;
        double i1 = 0.0, i2 = 0.0, j1 = 0.0, j2 = 0.0, s1 = 0.0, s2 = 0.0;
#pragma unroll
        for (int n = 27; n >= 2; --n) {
            const double nn = n;
            const double a0 = (nn + 2.0) / (nn + 1.0);
            const double r2 = 1.0 / (nn + 2.0);
            const double cb = (1.0 - 2.0 * (nn + 2.0)) / (2.0 * (nn + 2.0));
            const double sbp = ((n + 1) % 2 == 0) ? 1.0 : -1.0;
            const double in = a0 * ic * (ue * r2 - sbp * ub * r2 + cb * b * i1 - i2);
            const double jn = ic * (in - b * j1 - j2);
            const double sn = ic * (jn - b * s1 - s2);
            if (n < K) { I[n] = in; J[n] = jn; S[n] = sn; }
            i2 = i1; i1 = in; j2 = j1; j1 = jn; s2 = s1; s1 = sn;
        }
    }
}

// Near-pair buffer: per pair and source weight m = 1..N a 64-float record
// (16-byte aligned): the block columns 3(m-1)..3(m-1)+2 [col][row] (9N
// floats), then the velocity panel entries [w][col][a] (18 floats).
constexpr int kNearWeight = 64;
constexpr int kNearBlock = 5 * kNearWeight;
static_assert(9 * 5 + 18 <= kNearWeight, "near record");

// ---------------------------------------------------------------- classify
constexpr int kClassifyWarps = 4;

// One warp per target: the near-pair bitmap, the number of near sources before
// each bitmap word, the near sources in ascending order and their count, and
// the target's first slot in the near-pair buffer (claimed with an atomic add;
// slots only place the blocks, they do not change any value).
__global__ void __launch_bounds__(kClassifyWarps * 32) classify_kernel(SplitArgs a) {
    __shared__ double s_pv[kMaxLQ];
    for (int t = threadIdx.x; t < kMaxLQ; t += blockDim.x) s_pv[t] = t < a.LQ ? a.tab->pv[t] : 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * kClassifyWarps + warp;
    if (i >= a.M) return;  // whole warp
    const double xi0 = a.pos[3 * i], xi1 = a.pos[3 * i + 1], xi2 = a.pos[3 * i + 2];
    const double ti0 = a.ori[3 * i], ti1 = a.ori[3 * i + 1], ti2 = a.ori[3 * i + 2];
    int count = 0;
    int *list = a.near_list + (int64_t)i * a.M;
    for (int jw = 0; jw < a.words; ++jw) {
        const int j = jw * 32 + lane;
        bool near = false;
        if (j < a.M && j != i) {
            const double D0 = xi0 - a.pos[3 * j], D1 = xi1 - a.pos[3 * j + 1], D2 = xi2 - a.pos[3 * j + 2];
            for (int q = 0; q < a.LQ && !near; ++q) {
                const double s = s_pv[q];
                const double r0 = D0 + s * ti0, r1 = D1 + s * ti1, r2 = D2 + s * ti2;
                const double c = r0 * r0 + r1 * r1 + r2 * r2;
                near = c < a.near_c;
            }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, near);
        if (lane == 0) {
            a.near_bits[(int64_t)i * a.words + jw] = mask;
            a.near_pref[(int64_t)i * a.words + jw] = count;
        }
        if (near) list[count + __popc(mask & ((1u << lane) - 1u))] = j;
        count += __popc(mask);
    }
    if (lane == 0) {
        a.near_cnt[i] = count;
        a.near_off[i] = atomicAdd(a.near_total, count);
    }
}

// ---------------------------------------------------------------- far pairs (FP32)
// One warp per CTA; lane = target fiber, the warp walks a chunk of sources.
// For source weight m the block entries follow from
//   theta = AI I + D X^T + t Y^T + p Z^T,   X = R0 D + R1 t + C0 p,
//   Y = R1 D + R2 t + C1 p,  Z = C0 D + C1 t + E p,
//   Q = theta t = AI t + (D.t) X + (t.t) Y + (p.t) Z,
// the pair tensors of the header expanded.  The m loop runs at run time with
// the Legendre coefficients sc_m a_mp in constant memory, which keeps the
// kernel small enough for the instruction cache.

#define RF_LEG(m, p) ((float)(leg_scale(m) * leg_coef(m, p)))
#define RF_LEG_ROW(m) RF_LEG(m, 0), RF_LEG(m, 1), RF_LEG(m, 2), RF_LEG(m, 3), RF_LEG(m, 4), RF_LEG(m, 5), RF_LEG(m, 6), RF_LEG(m, 7)
__constant__ float c_leg32[8][8] = {{RF_LEG_ROW(0)}, {RF_LEG_ROW(1)}, {RF_LEG_ROW(2)}, {RF_LEG_ROW(3)},
                                    {RF_LEG_ROW(4)}, {RF_LEG_ROW(5)}, {RF_LEG_ROW(6)}, {RF_LEG_ROW(7)}};
#undef RF_LEG_ROW
#undef RF_LEG

#ifndef RF_FAR_MINB
#define RF_FAR_MINB 8
#endif
// Warps per far-pair CTA.  Each warp works on its own 32 targets; the warps
// of a CTA step through the sources together (a barrier before each source's
// post-processing), so the warps sharing a scheduler mostly run the same code
// at the same time and share the instruction cache: the Gauss-point loop and
// the post-processing together exceed it, and warps of separate one-warp CTAs
// drift into different phases.  Measured at M = 4000: assembly 20.35 ms with
// one-warp CTAs, 19.5 ms with barriers before both phases, 19.35 ms with the
// one before the post-processing alone.
#ifndef RF_FAR_WARPS
#define RF_FAR_WARPS 8
#endif

template <int N, bool PANELS>
struct FarSmem {
    static constexpr int GR = 32 * 3 * N;                   // staged rows of one column
    static constexpr int PAN = 2 * 3 * 96;                  // staged panel columns
    static constexpr int STG16 = 3 * GR / 2;                // BF16 copy (split storage: low plane) of the staged columns
    static constexpr size_t kBytes = sizeof(float) * (32 * kNearWeight + 16 + 64 + kMaxLQ +
                                                      kMaxLQ * SplitDims<N>::KWP + 3 * GR + (PANELS ? PAN : 0) +
                                                      STG16);
    static_assert(kBytes % 16 == 0, "each warp's region starts on a 16-byte boundary");
    static size_t bytes() { return kBytes; }
};

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
// Bulk asynchronous shared -> global copies (the copy engine streams staged
// columns out while the warp goes on computing).  Addresses and sizes are
// multiples of 16 bytes.
__device__ __forceinline__ void bulk_s2g(void *gdst, const void *ssrc, unsigned bytes) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(ssrc);
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(gdst), "r"(s), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
// lanes of a far-pair warp that hand staged column segments to the copy engine
constexpr int kCopyLanes = 12;
// the staged data has been read out: the staging buffers may be rewritten
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }
// generic-proxy shared-memory writes made visible to the bulk copies
__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

template <int N, bool PANELS>
__device__ __forceinline__ void far_store_m(const SplitArgs &a, int m, int j, int i0, int nvalid, const float *stg,
                                            const float *pan, __nv_bfloat16 *stg16, int lane) {
    constexpr int RB = 3 * N, GR = 32 * RB;
    const int64_t row0 = (int64_t)i0 * RB;
    const int nrows = nvalid * RB;
    const int64_t col0 = (int64_t)j * RB + 3 * (m - 1);
    if (nrows == GR) {
        // whole column segments: the 16-bit planes (or the BF16 copy) are
        // staged too, then one lane hands every segment to the copy engine
        // (the matrix: 3 x 32 targets x 3N rows; panels: 2 x 3 x 96 rows),
        // and the warp moves on
        if (a.A16lo) {
            // split FP32 storage: the low plane goes to the BF16 staging, the
            // high plane over the first half of the FP32 staging it is read
            // from (a step's writes reach only entries read by earlier steps
            // or, behind the barrier, by this one).  (u + 0x8000) >> 16 is
            // split_hi(u); the byte permutes pack two 16-bit halves.
            const uint4 *s4 = reinterpret_cast<const uint4 *>(stg);
            uint2 *dh = reinterpret_cast<uint2 *>(const_cast<float *>(stg));
            uint2 *dl = reinterpret_cast<uint2 *>(stg16);
            for (int e0 = 0; e0 < 3 * GR / 4; e0 += 32) {
                const int e = e0 + lane;
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (e < 3 * GR / 4) v = s4[e];
                __syncwarp();
                if (e < 3 * GR / 4) {
                    dh[e] = make_uint2(__byte_perm(v.x + 0x8000u, v.y + 0x8000u, 0x7632),
                                       __byte_perm(v.z + 0x8000u, v.w + 0x8000u, 0x7632));
                    dl[e] = make_uint2(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.z, v.w, 0x5410));
                }
            }
        } else if (a.A16) {
            const float4 *s4 = reinterpret_cast<const float4 *>(stg);
            uint2 *d2 = reinterpret_cast<uint2 *>(stg16);
            for (int e = lane; e < 3 * GR / 4; e += 32) {
                const float4 v = s4[e];
                __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                uint2 u;
                u.x = *reinterpret_cast<unsigned *>(&lo);
                u.y = *reinterpret_cast<unsigned *>(&hi);
                d2[e] = u;
            }
        }
        fence_async_shared();
        __syncwarp();
        // one segment per lane: lane l copies column bb = l % 3 of kind l / 3
        // (0: the FP32 words or the high plane, 1: the low plane or the BF16
        // copy, 2 and 3: the two panels); each lane commits its own group
        if (lane < kCopyLanes) {
            const int bb = lane % 3, kind = lane / 3;
            const int64_t col = col0 + bb;
            if (kind == 0) {
                if (a.A32)
                    bulk_s2g(a.A32 + col * a.lda + row0, stg + bb * GR, GR * sizeof(float));
                else if (a.A16lo)
                    bulk_s2g(a.A16 + col * a.lda + row0, reinterpret_cast<const unsigned short *>(stg) + bb * GR,
                             GR * sizeof(unsigned short));
            } else if (kind == 1) {
                if (a.A16lo)
                    bulk_s2g(a.A16lo + col * a.lda + row0, reinterpret_cast<const unsigned short *>(stg16) + bb * GR,
                             GR * sizeof(unsigned short));
                else if (a.A16)
                    bulk_s2g(a.A16 + col * a.lda + row0, stg16 + bb * GR, GR * sizeof(__nv_bfloat16));
            } else if (PANELS) {
                const int w = kind - 2;
                bulk_s2g((w ? a.PW32 : a.PV32) + col * a.ldp + (int64_t)i0 * 3, pan + (w * 3 + bb) * 96,
                         96 * sizeof(float));
            }
            bulk_commit();
        }
        return;
    }
#pragma unroll
    for (int bb = 0; bb < 3; ++bb) {
        const int64_t col = col0 + bb;
        const float *src = stg + bb * GR;
        for (int e = lane; e < nrows; e += 32) {
            const int64_t idx = col * a.lda + row0 + e;
            if (a.A16lo) {
                split_store(src[e], a.A16 + idx, a.A16lo + idx);
            } else {
                if (a.A32) a.A32[idx] = src[e];
                if (a.A16) a.A16[idx] = __float2bfloat16_rn(src[e]);
            }
        }
        if (PANELS) {
            const int prow = 3 * nvalid;
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                float *dst = (w ? a.PW32 : a.PV32) + col * a.ldp + (int64_t)i0 * 3;
                const float *ps = pan + (w * 3 + bb) * 96;
                for (int e = lane; e < prow; e += 32) dst[e] = ps[e];
            }
        }
    }
}

// Coefficient sets of weight m (parity PAR) for rows k = 0..N in registers:
// S[0..6][k] = AI, R0, R1, R2, C0, C1, E.
template <int N, int PAR>
__device__ __forceinline__ void far_sets_reg(int m, const float (&U)[N + 1][N + 1], const float (&V)[N + 3][N + 3],
                                             float (&S)[7][N + 1]) {
    constexpr int NP = (N - PAR) / 2 + 1;
    float cf[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) cf[i] = c_leg32[m][PAR + 2 * i];
    float R0[N + 3], C0[N + 2], R1[N + 2];
#pragma unroll
    for (int k = 0; k < N + 3; ++k) {
        float s1 = 0.f;
#pragma unroll
        for (int i = 0; i < NP; ++i) s1 = fmaf(cf[i], V[PAR + 2 * i][k], s1);
        R0[k] = s1;
    }
#pragma unroll
    for (int k = 0; k < N + 2; ++k) {
        float s1 = 0.f;
#pragma unroll
        for (int i = 0; i < NP; ++i)
            if (k < vrows(N, PAR + 2 * i + 1)) s1 = fmaf(cf[i], V[PAR + 2 * i + 1][k], s1);
        C0[k] = -s1;
    }
#pragma unroll
    for (int k = 0; k < N + 2; ++k)
        R1[k] = (float)bonnet_a(k) * R0[k + 1] + (k > 0 ? (float)bonnet_b(k) * R0[k > 0 ? k - 1 : 0] : 0.f);
#pragma unroll
    for (int k = 0; k <= N; ++k) {
        float ai = 0.f, ee = 0.f;
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            ai = fmaf(cf[i], U[PAR + 2 * i][k], ai);
            ee = fmaf(cf[i], V[PAR + 2 * i + 2][k], ee);
        }
        S[0][k] = ai;
        S[1][k] = R0[k];
        S[2][k] = R1[k];
        S[3][k] = (float)bonnet_a(k) * R1[k + 1] + (k > 0 ? (float)bonnet_b(k) * R1[k > 0 ? k - 1 : 0] : 0.f);
        S[4][k] = C0[k];
        S[5][k] = (float)bonnet_a(k) * C0[k + 1] + (k > 0 ? (float)bonnet_b(k) * C0[k > 0 ? k - 1 : 0] : 0.f);
        S[6][k] = ee;
    }
}

// A 3-vector with components 0 and 1 packed for the paired FP32 units.
struct V3p {
    float2 xy;
    float z;
};
__device__ __forceinline__ V3p v3p(const float *v) { return {make_float2(v[0], v[1]), v[2]}; }
__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }
// a A + b B + c C
__device__ __forceinline__ V3p comb3(float a, const V3p &A, float b, const V3p &B, float c, const V3p &C) {
    V3p r;
    r.xy = __ffma2_rn(dup2(c), C.xy, __ffma2_rn(dup2(b), B.xy, __fmul2_rn(dup2(a), A.xy)));
    r.z = fmaf(c, C.z, fmaf(b, B.z, a * A.z));
    return r;
}
// a A + b B + c C + d E
__device__ __forceinline__ V3p comb4(float a, const V3p &A, float b, const V3p &B, float c, const V3p &C, float d,
                                     const V3p &E) {
    V3p r;
    r.xy = __ffma2_rn(dup2(d), E.xy,
                      __ffma2_rn(dup2(c), C.xy, __ffma2_rn(dup2(b), B.xy, __fmul2_rn(dup2(a), A.xy))));
    r.z = fmaf(d, E.z, fmaf(c, C.z, fmaf(b, B.z, a * A.z)));
    return r;
}

// X = R0 D + R1 t + C0 p, Y = R1 D + R2 t + C1 p, Z = C0 D + C1 t + E p for row k
template <int N>
__device__ __forceinline__ void far_xyz_p(const float (&S)[7][N + 1], int k, const V3p &D, const V3p &t,
                                          const V3p &p, V3p &X, V3p &Y, V3p &Z) {
    const float R0 = S[1][k], R1 = S[2][k], R2 = S[3][k], C0 = S[4][k], C1 = S[5][k], E = S[6][k];
    X = comb3(R0, D, R1, t, C0, p);
    Y = comb3(R1, D, R2, t, C1, p);
    Z = comb3(C0, D, C1, t, E, p);
}

// The 3 x 3 entries sc (AI delta_ab + D_a X_b + t_a Y_b + p_a Z_b) at
// dst[b * ld + a]; columns b = 0, 1 as a packed pair.
__device__ __forceinline__ void block3(float *dst, int ld, float sc, float AI, const float *D, const float *t,
                                       const float *p, const V3p &X, const V3p &Y, const V3p &Z) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float2 d0 = make_float2(a == 0 ? AI : 0.f, a == 1 ? AI : 0.f);
        float2 e = __ffma2_rn(dup2(p[a]), Z.xy, __ffma2_rn(dup2(t[a]), Y.xy, __ffma2_rn(dup2(D[a]), X.xy, d0)));
        e = __fmul2_rn(dup2(sc), e);
        dst[a] = e.x;
        dst[ld + a] = e.y;
        dst[2 * ld + a] = sc * fmaf(p[a], Z.z, fmaf(t[a], Y.z, fmaf(D[a], X.z, a == 2 ? AI : 0.f)));
    }
}


template <int N, bool PANELS, bool FAR>
__global__ void __launch_bounds__(32 * RF_FAR_WARPS, RF_FAR_MINB / RF_FAR_WARPS) far_pairs_kernel(SplitArgs a) {
    using SD = SplitDims<N>;
    using SM = FarSmem<N, PANELS>;
    constexpr int NL = SD::NL, NV = SD::NV, KW = SD::KW, NRHS = SD::NRHS, RB = SD::RB, GR = SM::GR;
    extern __shared__ __align__(16) unsigned char smem_all[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *smem_raw = smem_all + (size_t)warp * SM::kBytes;  // this warp's region
    float *s_nb = reinterpret_cast<float *>(smem_raw);               // [near lane][kNearWeight], one weight
    float *s_gk = s_nb + 32 * kNearWeight;                            // gamma_k (0..7), E_k (8..15)
    int *s_nl = reinterpret_cast<int *>(s_gk + 16);                   // near lanes of the source, in order
    int *s_ns = s_nl + 32;                                            // and their buffer slots
    float *s_pv = reinterpret_cast<float *>(s_ns + 32);
    float *s_w = s_pv + kMaxLQ;                                       // [kMaxLQ][KWP]: w_q P_k(s_q), k >= KW zero
    float *s_stg = s_w + kMaxLQ * SD::KWP;                            // [3][GR]
    float *s_pan = s_stg + 3 * GR;                                    // [2][3][96]
    __nv_bfloat16 *s_stg16 = reinterpret_cast<__nv_bfloat16 *>(s_pan + (PANELS ? SM::PAN : 0));  // [3][GR]

    const Tables &tab = *a.tab;
    const int LQ = a.LQ;
    for (int t = lane; t < kMaxLQ; t += 32) s_pv[t] = t < LQ ? (float)tab.pv[t] : 0.f;
    for (int t = lane; t < kMaxLQ * SD::KWP; t += 32) {
        const int q = t / SD::KWP, k = t - q * SD::KWP;
        s_w[t] = (q < LQ && k < KW) ? (float)(tab.wv[q] * tab.P[k][q]) : 0.f;
    }
    if (lane < 8) {
        s_gk[lane] = lane <= N ? (float)tab.gamma[lane] : 0.f;
        s_gk[8 + lane] = lane <= N ? (float)tab.Ek[lane] : 0.f;
    }
    double rhs[NRHS];  // sum over the far sources of theta^k_0 f
#pragma unroll
    for (int r = 0; r < NRHS; ++r) rhs[r] = 0.0;
    __syncwarp();

    const float D1 = (float)tab.D1, sv = (float)(0.5 / tab.d), sw = (float)(1.5 / tab.d);
    const float f[3] = {(float)tab.half_force[0], (float)tab.half_force[1], (float)tab.half_force[2]};
    const float e2 = (float)(2.0 * tab.eps2), e6 = (float)(6.0 * tab.eps2);

    const int i0 = (blockIdx.x * RF_FAR_WARPS + warp) * 32;
    const int i = i0 + lane;
    const bool valid = i < a.M;
    const int nvalid = min(32, a.M - i0);     // <= 0 for a warp past the last target: it only keeps step
    const int ic = valid ? i : min(i0, a.M - 1);
    const double xi0 = a.pos[3 * ic], xi1 = a.pos[3 * ic + 1], xi2 = a.pos[3 * ic + 2];
    const float t[3] = {(float)a.ori[3 * ic], (float)a.ori[3 * ic + 1], (float)a.ori[3 * ic + 2]};
    const float tt = t[0] * t[0] + t[1] * t[1] + t[2] * t[2];
    const int64_t brow = (int64_t)ic * a.words;
    const int slot0 = (valid && a.near_bits) ? a.near_off[ic] : 0;
    const bool merge = a.near_bits != nullptr && a.merge != 0;

    const int j0 = blockIdx.y * a.chunk;
    const int j1 = min(a.M, j0 + a.chunk);
    // the source's centre and direction are loaded one source ahead
    double xj[3] = {0.0, 0.0, 0.0};
    float pj[3] = {0.f, 0.f, 0.f};
    if (j0 < j1) {
        xj[0] = __ldg(a.pos + 3 * j0); xj[1] = __ldg(a.pos + 3 * j0 + 1); xj[2] = __ldg(a.pos + 3 * j0 + 2);
        pj[0] = (float)__ldg(a.ori + 3 * j0); pj[1] = (float)__ldg(a.ori + 3 * j0 + 1); pj[2] = (float)__ldg(a.ori + 3 * j0 + 2);
    }
    // staging offsets of this thread's entries in a near record: block entries
    // e = lane and lane + 32 (e = 3 RB columns-major), panel entry lane < 18
    const int moff0 = (lane / RB) * GR + lane % RB;
    const int moff1 = ((lane + 32) / RB) * GR + (lane + 32) % RB;
    const int poff = 3 * GR + ((lane / 9) * 3 + (lane % 9) / 3) * 96 + (lane % 9) % 3;  // s_pan follows s_stg
    unsigned word = 0u;
    int wpref = 0;
    for (int j = j0; j < j1; ++j) {
        const float D[3] = {(float)(xi0 - xj[0]), (float)(xi1 - xj[1]), (float)(xi2 - xj[2])};
        const float p[3] = {pj[0], pj[1], pj[2]};
        if (j + 1 < j1) {
            xj[0] = __ldg(a.pos + 3 * j + 3); xj[1] = __ldg(a.pos + 3 * j + 4); xj[2] = __ldg(a.pos + 3 * j + 5);
            pj[0] = (float)__ldg(a.ori + 3 * j + 3); pj[1] = (float)__ldg(a.ori + 3 * j + 4); pj[2] = (float)__ldg(a.ori + 3 * j + 5);
        }
        bool near = false;
        int slot = 0;
        if (valid && a.near_bits) {
            if (j == j0 || (j & 31) == 0) {
                word = a.near_bits[brow + (j >> 5)];
                wpref = merge ? a.near_pref[brow + (j >> 5)] : 0;
            }
            near = (word >> (j & 31)) & 1u;
            if (near) slot = slot0 + wpref + __popc(word & ((1u << (j & 31)) - 1u));
        }
        const unsigned nmask = merge ? __ballot_sync(0xffffffffu, near) : 0u;
        const int nnear = __popc(nmask);
        // list the near lanes in order and prefetch their weight-1 records;
        // the Gauss-point loop hides the copy
        if (near && merge) {
            const int r = __popc(nmask & ((1u << lane) - 1u));
            s_nl[r] = lane;
            s_ns[r] = slot;
        }
        __syncwarp();
        for (int u = lane; u < nnear * (kNearWeight / 4); u += 32) {
            const int r = u >> 4, c = u & 15;  // kNearWeight / 4 = 16 chunks per record
            cp_async16(s_nb + r * kNearWeight + 4 * c, a.nearbuf + (int64_t)s_ns[r] * kNearBlock + 4 * c);
        }
        cp_async_commit();
        const bool diag = i == j;
        const bool act = valid && !near && !diag;

        float U[NL][NL], V[NV][KW];
#pragma unroll
        for (int pp = 0; pp < NL; ++pp)
#pragma unroll
            for (int k = 0; k < NL; ++k) U[pp][k] = 0.f;
#pragma unroll
        for (int pp = 0; pp < NV; ++pp)
#pragma unroll
            for (int k = 0; k < KW; ++k) V[pp][k] = 0.f;
        // the Gauss point q's moments, weighted, into the projections
        // Pairs of rows (k, k + 1) go through the packed FP32 units: each half
        // of __ffma2_rn is the fmaf of the scalar form, so the sums are the same.
        auto add_point = [&](int q, const float *I, const float *J, const float *S) {
            constexpr int KWP = SD::KWP;
            const float2 *w2 = reinterpret_cast<const float2 *>(s_w + q * KWP);  // even stride: 8-byte aligned
            float2 wk[KWP / 2];
#pragma unroll
            for (int k = 0; k < KWP / 2; ++k) wk[k] = w2[k];
#pragma unroll
            for (int pp = 0; pp < NL; ++pp) {
                const float u = fmaf(e2, J[pp], I[pp]);
                const float2 u2 = make_float2(u, u);
#pragma unroll
                for (int k = 0; k + 1 < NL; k += 2) {
                    const float2 r = __ffma2_rn(wk[k / 2], u2, make_float2(U[pp][k], U[pp][k + 1]));
                    U[pp][k] = r.x;
                    U[pp][k + 1] = r.y;
                }
                if (NL % 2) U[pp][NL - 1] = fmaf(wk[(NL - 1) / 2].x, u, U[pp][NL - 1]);
            }
#pragma unroll
            for (int pp = 0; pp < NV; ++pp) {
                const float v = fmaf(-e6, S[pp], J[pp]);
                const float2 v2 = make_float2(v, v);
#pragma unroll
                for (int k = 0; k < KW; k += 2) {
                    if (k + 1 < vrows(N, pp)) {
                        const float2 r = __ffma2_rn(wk[k / 2], v2, make_float2(V[pp][k], V[pp][k + 1]));
                        V[pp][k] = r.x;
                        V[pp][k + 1] = r.y;
                    } else if (k < vrows(N, pp)) {
                        V[pp][k] = fmaf(wk[k / 2].x, v, V[pp][k]);
                    }
                }
            }
        };
        if (act) {
            if constexpr (FAR) {
                // every point far (c >= 6): two Gauss points per pass of the
                // packed recursion, added in the order q, q + 1.  Past an odd LQ
                // the partner is the zero padding of s_pv: computed, not added.
                static_assert(kMaxLQ % 2 == 0, "the partner of the last point must lie in s_pv");
                for (int q = 0; q < LQ; q += 2) {
                    const float sa = s_pv[q], sb = s_pv[q + 1];
                    const Geom32 ga(fmaf(sa, t[0], D[0]), fmaf(sa, t[1], D[1]), fmaf(sa, t[2], D[2]), p[0], p[1], p[2]);
                    const Geom32 gb(fmaf(sb, t[0], D[0]), fmaf(sb, t[1], D[1]), fmaf(sb, t[2], D[2]), p[0], p[1], p[2]);
                    float2 I2[KW], J2[KW], S2[KW];
                    moments_backward_fp32x2<N>(make_float2(ga.b, gb.b), make_float2(ga.c, gb.c), I2, J2, S2);
                    float I[KW], J[KW], S[KW];
#pragma unroll
                    for (int k = 0; k < KW; ++k) { I[k] = I2[k].x; J[k] = J2[k].x; S[k] = S2[k].x; }
                    add_point(q, I, J, S);
                    if (q + 1 < LQ) {
#pragma unroll
                        for (int k = 0; k < KW; ++k) { I[k] = I2[k].y; J[k] = J2[k].y; S[k] = S2[k].y; }
                        add_point(q + 1, I, J, S);
                    }
                }
            } else {
                // two Gauss points in flight (two independent recursions): 2 % faster
                // once the warps of a scheduler share the instruction stream
#pragma unroll 2
                for (int q = 0; q < LQ; ++q) {
                    const float sq = s_pv[q];
                    const float r0x = fmaf(sq, t[0], D[0]), r0y = fmaf(sq, t[1], D[1]), r0z = fmaf(sq, t[2], D[2]);
                    float I[KW], J[KW], S[KW];
                    moments_fp32<N, FAR>(Geom32(r0x, r0y, r0z, p[0], p[1], p[2]), I, J, S);
                    add_point(q, I, J, S);
                }
            }
        }
        const float Dt = D[0] * t[0] + D[1] * t[1] + D[2] * t[2];
        const float pt = p[0] * t[0] + p[1] * t[1] + p[2] * t[2];
        cp_async_wait_all();
        __syncthreads();  // the CTA's warps enter each source's post-processing together

        if (act) {
            // right-hand side: theta^k_0 f for weight 0 (near pairs add theirs in the near kernel)
#pragma unroll
            for (int k = 0; k <= N; ++k) {
                float R0[3] = {0.f, 0.f, 0.f}, C0[3] = {0.f, 0.f, 0.f};
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    const int kk = k - 1 + o;
                    if (kk >= 0) C0[o] = -V[1][kk];
                }
                const float AI = U[0][k], E = V[2][k];
                const float R0k = V[0][k], R0p = V[0][k + 1], R0pp = V[0][k + 2];
                const float R0m = k > 0 ? V[0][k > 0 ? k - 1 : 0] : 0.f, R0mm = k > 1 ? V[0][k > 1 ? k - 2 : 0] : 0.f;
                const float R1 = (float)bonnet_a(k) * R0p + (float)bonnet_b(k) * R0m;
                const float R1p = (float)bonnet_a(k + 1) * R0pp + (float)bonnet_b(k + 1) * R0k;
                const float R1m = k > 0 ? (float)bonnet_a(k - 1) * R0k + (float)bonnet_b(k - 1) * R0mm : 0.f;
                const float R2 = (float)bonnet_a(k) * R1p + (float)bonnet_b(k) * R1m;
                const float C1 = (float)bonnet_a(k) * C0[2] + (float)bonnet_b(k) * C0[0];
                (void)R0;
                float X[3], Y[3], Z[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    X[c] = R0k * D[c] + R1 * t[c] + C0[1] * p[c];
                    Y[c] = R1 * D[c] + R2 * t[c] + C1 * p[c];
                    Z[c] = C0[1] * D[c] + C1 * t[c] + E * p[c];
                }
                const float Xf = X[0] * f[0] + X[1] * f[1] + X[2] * f[2];
                const float Yf = Y[0] * f[0] + Y[1] * f[1] + Y[2] * f[2];
                const float Zf = Z[0] * f[0] + Z[1] * f[1] + Z[2] * f[2];
#pragma unroll
                for (int c = 0; c < 3; ++c) rhs[3 * k + c] += (double)(AI * f[c] + D[c] * Xf + t[c] * Yf + p[c] * Zf);
            }
        }

        // weights m = 1..N: odd weights first, then even ones (sc_m a_mp vanishes
        // unless p and m have the same parity); the near records of the next
        // weight in this order are prefetched behind the current one
#pragma unroll 1
        for (int it = 0; it < N; ++it) {
            const int m = it < (N + 1) / 2 ? 2 * it + 1 : 2 * (it - (N + 1) / 2) + 2;
            float S[7][N + 1];
            if (m & 1) far_sets_reg<N, 1>(m, U, V, S);
            else far_sets_reg<N, 0>(m, U, V, S);
            // the block entries and panel rows: theta's 3 x 3 blocks with their
            // columns (components of X, Y, Z) paired on the packed FP32 units
            const V3p Dp = v3p(D), tp = v3p(t), pp3 = v3p(p);
            // the copy engine has read the previous weight's staged columns
            // (waited for only here, so that the coefficient sets above
            // overlap the copies)
            if (lane < kCopyLanes) bulk_wait_read();
            __syncwarp();
            // row k = 0: velocity panel P0 only
            if (PANELS) {
                V3p X, Y, Z;
                far_xyz_p<N>(S, 0, Dp, tp, pp3, X, Y, Z);
                block3(s_pan + lane * 3, 96, sv, S[0][0], D, t, p, X, Y, Z);
            }
            // row k = 1: block row D1 t (theta t)^T and velocity panel P1
            {
                V3p X, Y, Z;
                far_xyz_p<N>(S, 1, Dp, tp, pp3, X, Y, Z);
                const float AI = S[0][1];
                const V3p Q = comb4(AI, tp, Dt, X, tt, Y, pt, Z);
                const float Qv[3] = {Q.xy.x, Q.xy.y, Q.z};
#pragma unroll
                for (int bb = 0; bb < 3; ++bb)
#pragma unroll
                    for (int aa = 0; aa < 3; ++aa) s_stg[bb * GR + lane * RB + aa] = D1 * t[aa] * Qv[bb];
                if (PANELS) {
                    V3p YQ;
                    YQ.xy = make_float2(Y.xy.x - Q.xy.x, Y.xy.y - Q.xy.y);
                    YQ.z = Y.z - Q.z;
                    block3(s_pan + 3 * 96 + lane * 3, 96, sw, AI, D, t, p, X, YQ, Z);
                }
            }
            // rows k = 2..N: gamma_k (theta - E_k t (theta t)^T)
#pragma unroll
            for (int k = 2; k <= N; ++k) {
                V3p X, Y, Z;
                far_xyz_p<N>(S, k, Dp, tp, pp3, X, Y, Z);
                const float AI = S[0][k], g = s_gk[k], ek = s_gk[8 + k];
                const V3p Q = comb4(AI, tp, Dt, X, tt, Y, pt, Z);
                V3p W;
                W.xy = __ffma2_rn(dup2(-ek), Q.xy, Y.xy);
                W.z = fmaf(-ek, Q.z, Y.z);
                block3(s_stg + lane * RB + 3 * (k - 1), GR, g, AI, D, t, p, X, W, Z);
            }
            // the diagonal pair (its projections are zero): identity where k = m
            if (diag) {
#pragma unroll
                for (int aa = 0; aa < 3; ++aa) s_stg[aa * GR + lane * RB + 3 * (m - 1) + aa] = 1.f;
            }
            cp_async_wait_all();
            __syncwarp();
            // near pairs: the FP64-integrated columns of weight m replace the
            // staged zeros; entry offsets are fixed per thread
            for (int r = 0; r < nnear; ++r) {
                const int L = s_nl[r];
                const float *src = s_nb + r * kNearWeight;
                if (lane < 3 * RB) s_stg[moff0 + L * RB] = src[lane];
                if (lane < 3 * RB - 32) s_stg[moff1 + L * RB] = src[lane + 32];
                if (PANELS && lane < 18) s_stg[poff + L * 3] = src[3 * RB + lane];
            }
            __syncwarp();
            // the records of the next weight, hidden behind the stores and that weight's work
            if (it + 1 < N) {
                const int mn = it + 1 < (N + 1) / 2 ? 2 * it + 3 : 2 * (it + 1 - (N + 1) / 2) + 2;
                for (int u = lane; u < nnear * (kNearWeight / 4); u += 32) {
                    const int r = u >> 4, c = u & 15;
                    cp_async16(s_nb + r * kNearWeight + 4 * c,
                               a.nearbuf + (int64_t)s_ns[r] * kNearBlock + (mn - 1) * kNearWeight + 4 * c);
                }
                cp_async_commit();
            }
            far_store_m<N, PANELS>(a, m, j, i0, nvalid, s_stg, s_pan, s_stg16, lane);
            __syncwarp();
        }
    }
    if (valid) {
#pragma unroll
        for (int r = 0; r < NRHS; ++r) a.far_contr[((int64_t)blockIdx.y * a.M + i) * NRHS + r] = rhs[r];
    }
    if (lane < kCopyLanes) bulk_wait_all();  // every staged segment written before the CTA's shared memory goes
}

// ---------------------------------------------------------------- near pairs (FP64)
constexpr int kNearWarps = 4;
// A pair's staged record: weight stride 66 floats (even: the copy reads float2),
// so the 20 lanes (pair, m >= 1) that store an entry use 16 different banks
constexpr int kNearStage = kNearWeight + 2;

template <int N>
struct NearSmem {
    using D = Dims64<N>;
    static constexpr int NRHS = 3 * (N + 1);
    static constexpr int PAIR = N * kNearStage;                          // floats of a staged pair
    static constexpr int THS = (D::TH + 1) / 2 * 2 + kTI * PAIR / 2;     // projections, then the staged records
    static_assert(kTI * PAIR % 2 == 0, "staged records in doubles");
    // the scalars G, or what follows them
    __host__ __device__ static constexpr int region(int LQ) {
        return ((D::COLS * ldq_of(LQ) > THS ? D::COLS * ldq_of(LQ) : THS) + 1) / 2 * 2;
    }
    // region, 4 sources, the warp's right-hand-side sums, the point list
    __host__ __device__ static constexpr int warp(int LQ) {
        return region(LQ) + kTI * 6 + kTI * NRHS + kTI * kMaxLQ / 8;
    }
    static constexpr int TABLES = kMaxLQ + (N + 3) * (int)(sizeof(RowTab) / sizeof(double)) + 3 * (N + 1) + Far<N>::kCoef + 6;
    static size_t bytes(int LQ) { return sizeof(double) * (TABLES + 1 + (size_t)kNearWarps * warp(LQ)); }
};

// One CTA per target fiber; a warp takes four of its near sources at a time.
// The pairs' points are split into those of the backward recursion run to n = 0
// (far_point) and the rest, which keep the reference's closed forms, so that
// every warp pass runs one of the two; then projections on the FP64 tensor
// cores and the block rows as in assemble64.cu, lane = (pair, m).  The four
// records leave together, consecutive slots, to the near-pair buffer (direct =
// false; the far kernel merges them into its column stores) or straight into A
// (direct = true, used when the buffer could not be grown).
// Bound by FP64 and integer issue (53 % of the issue slots, FP64 pipe 46 %).  One
// warp per pair (24 of 32 lanes with a point, each running the 26-step backward
// recursion or the forward one, a 36-way division of the block over 32 lanes)
// took 2.19 ms for the 460 thousand near pairs of a cloud of 2000 fibers; four
// pairs per warp take 0.97 ms.
template <int N, bool PANELS, int KSMAX>
__global__ void __launch_bounds__(kNearWarps * 32, 4) near_pairs_kernel(SplitArgs a, int direct) {
    using D = Dims64<N>;
    using SM = NearSmem<N>;
    constexpr int NL = D::NL, NC = D::NC, NU = D::NU, KST = D::KST, RB = 3 * N, NRHS = SM::NRHS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int LQ = a.LQ, LDQ = ldq_of(LQ), KS = (LQ + 3) / 4;
    const Tables &tab = *a.tab;
    const int i = blockIdx.x;

    double *s_pv = reinterpret_cast<double *>(smem_raw);            // kMaxLQ
    RowTab *s_row = reinterpret_cast<RowTab *>(s_pv + kMaxLQ);       // NL block rows, then 2 panel rows
    double *s_leg = reinterpret_cast<double *>(s_row + NL + 2);      // NL x 3
    double *s_far = s_leg + NL * 3;                                  // Far<N>::kCoef
    double *s_x = s_far + Far<N>::kCoef;                             // target centre and direction
    double *s_warp = s_pv + (SM::TABLES + 1) / 2 * 2;                // 16-byte aligned
    double *s_wP = s_warp;                                           // 8 x kMaxLQ, until the operands are loaded
    double *s_g = s_warp + warp * SM::warp(LQ);
    double *s_th = s_g;                                              // after the projection
    float *s_rec = reinterpret_cast<float *>(s_th + (D::TH + 1) / 2 * 2);
    double *s_src = s_g + SM::region(LQ);                            // 4 x (x, t)
    double *s_acc = s_src + kTI * 6;                                 // 4 x NRHS
    unsigned char *s_list = reinterpret_cast<unsigned char *>(s_acc + kTI * NRHS);

    for (int t = tid; t < kMaxLQ; t += kNearWarps * 32) s_pv[t] = t < LQ ? tab.pv[t] : 0.0;
    for (int t = tid; t < 8 * kMaxLQ; t += kNearWarps * 32) {
        const int m = t / kMaxLQ, q = t % kMaxLQ;
        s_wP[t] = (m <= N + 2 && q < LQ) ? tab.wv[q] * tab.P[m][q] : 0.0;
    }
    block_tables<N>(tab, s_row, s_leg, tid);
    for (int t = tid; t < Far<N>::kCoef; t += kNearWarps * 32) s_far[t] = Far<N>::coef(t);
    if (tid < 6) s_x[tid] = tid < 3 ? a.pos[3 * i + tid] : a.ori[3 * i + tid - 3];
    __syncthreads();
    double afrag[KSMAX];
#pragma unroll
    for (int s = 0; s < KSMAX; ++s) afrag[s] = s < KS ? s_wP[(lane >> 2) * kMaxLQ + 4 * s + (lane & 3)] : 0.0;
    __syncthreads();

    const double eps2 = tab.eps2;
    const int cnt = a.near_cnt[i];
    const int *list = a.near_list + (int64_t)i * a.M;
    const int64_t slot0 = a.near_off[i];
    const int ti3 = lane / NL, m3 = lane - ti3 * NL;
    for (int e = lane; e < kTI * NRHS; e += 32) s_acc[e] = 0.0;

    auto point = [&](int item, double &b, double &c) {
        const int ti = item / LQ, q = item - ti * LQ;
        const double sq = s_pv[q];
        const double *y = s_src + ti * 6;
        const double r0x = (s_x[0] - y[0]) + sq * s_x[3], r0y = (s_x[1] - y[1]) + sq * s_x[4],
                     r0z = (s_x[2] - y[2]) + sq * s_x[5];
        b = -2.0 * (y[3] * r0x + y[4] * r0y + y[5] * r0z);
        c = r0x * r0x + r0y * r0y + r0z * r0z;
    };

    for (int s0 = warp * kTI; s0 < cnt; s0 += kNearWarps * kTI) {
        const int npair = min(kTI, cnt - s0);
        const int npts = npair * LQ;
        if (lane < kTI * 6) {
            const int ti = lane / 6, c = lane % 6;
            // an unused pair repeats the last one's source; its scalars are zero
            const int j = list[s0 + min(ti, npair - 1)];
            s_src[lane] = c < 3 ? a.pos[3 * j + c] : a.ori[3 * j + c - 3];
        }
        __syncwarp();
        // the points: far ones listed from the front, the others from the back
        int nfar = 0, nnear = 0;
#pragma unroll 1
        for (int base = 0; base < npts; base += 32) {
            const int item = base + lane;
            double b = 0.0, c = 1.0;
            if (item < npts) point(item, b, c);
            const bool far = item < npts && far_point(b, c), near = item < npts && !far;
            const unsigned mf = __ballot_sync(0xffffffffu, far), mn = __ballot_sync(0xffffffffu, near);
            const unsigned below = (1u << lane) - 1u;
            if (far) s_list[nfar + __popc(mf & below)] = (unsigned char)item;
            if (near) s_list[npts - 1 - nnear - __popc(mn & below)] = (unsigned char)item;
            nfar += __popc(mf);
            nnear += __popc(mn);
        }
        // unused pairs, and the points between LQ and the next multiple of 4, are zero
        if (npair < kTI)
            for (int t = lane; t < (kTI - npair) * NC * LDQ; t += 32) s_g[npair * NC * LDQ + t] = 0.0;
        const int pad = 4 * KS - LQ;
        for (int t = lane; t < D::COLS * pad; t += 32) s_g[(t / pad) * LDQ + LQ + t % pad] = 0.0;
        __syncwarp();
#pragma unroll 1
        for (int u = lane; u < nfar; u += 32) {
            const int item = s_list[u], ti = item / LQ;
            double b, c;
            point(item, b, c);
            moments_far_fp64<N>(b, c, eps2, s_far, GStoreUV{s_g + ti * NC * LDQ + item - ti * LQ, LDQ, NU});
        }
#pragma unroll 1
        for (int u = lane; u < nnear; u += 32) {
            const int item = s_list[npts - 1 - u], ti = item / LQ;
            double b, c, I[N + 3], J[N + 3], S[N + 3];
            point(item, b, c);
            moments_near<N>(b, c, I, J, S);
            double *g = s_g + ti * NC * LDQ + item - ti * LQ;
#pragma unroll
            for (int p = 0; p <= N; ++p) g[p * LDQ] = I[p] + 2.0 * eps2 * J[p];
#pragma unroll
            for (int p = 0; p <= N + 2; ++p) g[(NU + p) * LDQ] = J[p] - 6.0 * eps2 * S[p];
        }
        __syncwarp();
        project_pairs<N, KSMAX>(s_g, s_th, afrag, LDQ, KS, lane);
        if (ti3 < npair) {
            const double *y = s_src + ti3 * 6;
            float *rec = s_rec + ti3 * SM::PAIR + (m3 - 1) * kNearStage;
            double *acc = s_acc + ti3 * NRHS;
            const double f0 = tab.half_force[0], f1 = tab.half_force[1], f2 = tab.half_force[2];
            block_rows<N, true>(s_row, s_leg, s_th + ti3 * D::PST + m3 * KST, m3, s_x, y, y + 3,
                                [&](int k, const BlockRow &r) {
                if (m3 == 0) {  // theta^k_0 f
                    const double Xf = r.X0 * f0 + r.X1 * f1 + r.X2 * f2, Yf = r.Y0 * f0 + r.Y1 * f1 + r.Y2 * f2,
                                 Zf = r.Z0 * f0 + r.Z1 * f1 + r.Z2 * f2;
                    acc[3 * k] += r.AI * f0 + r.D0 * Xf + r.t0 * Yf + r.p0 * Zf;
                    acc[3 * k + 1] += r.AI * f1 + r.D1 * Xf + r.t1 * Yf + r.p1 * Zf;
                    acc[3 * k + 2] += r.AI * f2 + r.D2 * Xf + r.t2 * Yf + r.p2 * Zf;
                    return;
                }
                auto block = [&](const RowTab &rt, float *out, int ld) {
                    double v[9];
                    r.entries(rt.g1, rt.g2, v);
#pragma unroll
                    for (int e = 0; e < 9; ++e) out[(e / 3) * ld + e % 3] = (float)v[e];
                };
                if (k > 0) block(s_row[k], rec + 3 * (k - 1), RB);
                if (PANELS && k < 2) block(s_row[NL + k], rec + 3 * RB + 9 * k, 3);
            });
        }
        __syncwarp();
        if (!direct) {
            float2 *dst = reinterpret_cast<float2 *>(a.nearbuf + (slot0 + s0) * kNearBlock);
            for (int e = lane; e < npair * N * (kNearWeight / 2); e += 32) {
                const int r = e / (kNearWeight / 2), w = e % (kNearWeight / 2);  // r: (pair, weight)
                dst[(r / N) * (kNearBlock / 2) + (r % N) * (kNearWeight / 2) + w] =
                    *reinterpret_cast<const float2 *>(s_rec + r * kNearStage + 2 * w);
            }
        } else {
            for (int e = lane; e < npair * N * kNearWeight; e += 32) {
                const int pr = e / (N * kNearWeight), mm = e / kNearWeight - pr * N, r = e % kNearWeight;
                const int64_t j = list[s0 + pr];
                const float v = s_rec[pr * SM::PAIR + mm * kNearStage + r];
                if (r < 3 * RB) {
                    const int col = 3 * mm + r / RB, rr = r % RB;
                    const int64_t idx = (j * RB + col) * a.lda + (int64_t)i * RB + rr;
                    if (a.A16lo) {
                        split_store(v, a.A16 + idx, a.A16lo + idx);
                    } else {
                        if (a.A32) a.A32[idx] = v;
                        if (a.A16) a.A16[idx] = __float2bfloat16_rn(v);
                    }
                } else if (PANELS && r < 3 * RB + 18) {
                    const int e2 = r - 3 * RB, w = e2 / 9, rem = e2 - w * 9, bb = rem / 3, aa = rem - bb * 3;
                    (w ? a.PW32 : a.PV32)[(j * RB + 3 * mm + bb) * a.ldp + (int64_t)i * 3 + aa] = v;
                }
            }
        }
        __syncwarp();
    }
    __syncthreads();
    for (int r = tid; r < NRHS; r += kNearWarps * 32) {
        double s = 0.0;
        for (int w = 0; w < kNearWarps * kTI; ++w)
            s += (s_warp + (w / kTI) * SM::warp(LQ) + SM::region(LQ) + kTI * 6)[(w % kTI) * NRHS + r];
        a.near_contr[(int64_t)i * NRHS + r] = s;
    }
}

// ---------------------------------------------------------------- finish
// b rows and the l = 0 velocity terms from the summed theta^k_0 f
// (matrix_assembly.f90:874-899; coeffs_and_vels.f90:698-705 for the velocity).
// A warp per fiber, lane = (k, component): the chunks' sums of a fiber are
// consecutive, so a chunk is one coalesced load.  A thread per fiber, reading
// them one by one, took 194 us at M = 1000, 138 us at M = 2000; 34 and 24 us.
constexpr int kFinishWarps = 4;

__global__ void __launch_bounds__(32 * kFinishWarps) split_finish_kernel(SplitArgs a, int nchunks, double *b,
                                                                         double *vpart) {
    const int lane = threadIdx.x & 31, i = blockIdx.x * kFinishWarps + (threadIdx.x >> 5);
    if (i >= a.M) return;  // whole warp
    const int N = a.N, NRHS = 3 * (N + 1);  // N <= 5: at most 18 lanes
    const int k = lane / 3, aa = lane - 3 * k;
    const Tables &tab = *a.tab;
    double s = 0.0;
    if (lane < NRHS) {
        const double *p = a.far_contr + (int64_t)i * NRHS + lane;
#pragma unroll 8
        for (int ch = 0; ch < nchunks; ++ch) s += p[(int64_t)ch * a.M * NRHS];
        if (a.near_contr) s += a.near_contr[(int64_t)i * NRHS + lane];
    }
    const double c0 = __shfl_sync(0xffffffffu, s, (3 * k) & 31), c1 = __shfl_sync(0xffffffffu, s, (3 * k + 1) & 31),
                 c2 = __shfl_sync(0xffffffffu, s, (3 * k + 2) & 31);
    if (lane >= NRHS) return;
    const double *t = a.ori + 3 * i;
    const double tdc = t[0] * c0 + t[1] * c1 + t[2] * c2;
    if (k >= 1)
        b[(int64_t)i * 3 * N + 3 * (k - 1) + aa] =
            (k == 1) ? -tab.D1 * tdc * t[aa] : -tab.gamma[k] * (s - tab.Ek[k] * tdc * t[aa]);
    if (vpart && k == 0) vpart[(int64_t)i * 6 + aa] = 0.5 / tab.d * s;
    if (vpart && k == 1) vpart[(int64_t)i * 6 + 3 + aa] = 1.5 / tab.d * (s - tdc * t[aa]);
}

template <int N, bool PANELS, bool FAR>
cudaError_t launch_far_n(const SplitArgs &a, int far_chunks, cudaStream_t st) {
    const size_t smem = RF_FAR_WARPS * FarSmem<N, PANELS>::bytes();
    auto kern = far_pairs_kernel<N, PANELS, FAR>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    const int groups = (a.M + 31) / 32;
    dim3 grid((groups + RF_FAR_WARPS - 1) / RF_FAR_WARPS, far_chunks);
    kern<<<grid, 32 * RF_FAR_WARPS, smem, st>>>(a);
    return cudaGetLastError();
}

template <int N, bool PANELS>
cudaError_t launch_near_n(const SplitArgs &a, bool direct, cudaStream_t st) {
    const size_t smem = NearSmem<N>::bytes(a.LQ);
    // tensor-core k-steps: 6 cover the usual 24 points
    auto kern = a.LQ <= 24 ? near_pairs_kernel<N, PANELS, 6> : near_pairs_kernel<N, PANELS, kMaxLQ / 4>;
    cudaError_t err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    kern<<<a.M, kNearWarps * 32, smem, st>>>(a, direct);
    return cudaGetLastError();
}

}  // namespace

// N <= 5: the near kernel projects onto P_0..P_{N+2} with one 8-row tensor-core tile
bool split_supported(int N, int LQ) { return N >= 1 && N <= 5 && LQ <= kMaxLQ; }

int split_far_chunks(int M, int sm_count) {
    const int groups = (M + 31) / 32;
    const int ctas_x = (groups + RF_FAR_WARPS - 1) / RF_FAR_WARPS;
    // a first guess: about 64 target groups' worth of CTAs per SM
    const int c0 = std::max(1, std::min((sm_count * 64 + groups - 1) / groups, M));
    const int per0 = (M + c0 - 1) / c0;
    // The CTAs (one per SM: registers) run in rounds of sm_count, each CTA
    // taking time in proportion to its sources, so the kernel takes about
    // rounds x sources per CTA: the sources per CTA within a factor 2 of the
    // guess that minimise that product (ties: the larger share, fewer CTAs).
    // At M = 4000 on 148 SMs: 87 sources per CTA, 736 CTAs in 4.97 rounds,
    // instead of 53 sources and 1216 CTAs in 8.2 rounds (17.06 -> 15.92 ms
    // per mixed assembly, the same matrix).
    int best_cost = -1, best_chunks = c0, best_per = per0;
    for (int per = std::max(1, per0 / 2); per <= 2 * per0 && per <= M; ++per) {
        const int chunks = (M + per - 1) / per;
        const int share = (M + chunks - 1) / chunks;
        const int64_t rounds = ((int64_t)ctas_x * chunks + sm_count - 1) / sm_count;
        const int64_t cost = rounds * share;
        if (best_cost < 0 || cost < best_cost || (cost == best_cost && share > best_per)) {
            best_cost = (int)cost;
            best_chunks = chunks;
            best_per = share;
        }
    }
    return std::max(1, std::min(best_chunks, M));
}

cudaError_t launch_split_classify(const SplitArgs &a, cudaStream_t st) {
    cudaError_t err = cudaMemsetAsync(a.near_total, 0, sizeof(int), st);
    if (err != cudaSuccess) return err;
    classify_kernel<<<(a.M + kClassifyWarps - 1) / kClassifyWarps, kClassifyWarps * 32, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_split_far(const SplitArgs &a, int far_chunks, cudaStream_t st) {
    const bool panels = a.PV32 != nullptr;
    // far pairs have c >= near_c >= kSplitMinNearC at every point: the FP32
    // backward recursion alone covers them
    const bool far_only = a.near_bits != nullptr && a.near_c >= kSplitMinNearC;
    switch (a.N) {
#define RF_FAR_CASE(n)                                                                                     \
    case n:                                                                                                \
        if (panels) return far_only ? launch_far_n<n, true, true>(a, far_chunks, st)                       \
                                    : launch_far_n<n, true, false>(a, far_chunks, st);                     \
        return far_only ? launch_far_n<n, false, true>(a, far_chunks, st)                                  \
                        : launch_far_n<n, false, false>(a, far_chunks, st);
        RF_FAR_CASE(1)
        RF_FAR_CASE(2)
        RF_FAR_CASE(3)
        RF_FAR_CASE(4)
        RF_FAR_CASE(5)
#undef RF_FAR_CASE
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_split_near(const SplitArgs &a, bool direct, cudaStream_t st) {
    const bool panels = a.PV32 != nullptr;
    switch (a.N) {
#define RF_NEAR_CASE(n) \
    case n: return panels ? launch_near_n<n, true>(a, direct, st) : launch_near_n<n, false>(a, direct, st);
        RF_NEAR_CASE(1)
        RF_NEAR_CASE(2)
        RF_NEAR_CASE(3)
        RF_NEAR_CASE(4)
        RF_NEAR_CASE(5)
#undef RF_NEAR_CASE
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_split_finish(const SplitArgs &a, int far_chunks, double *b, double *vpart, cudaStream_t st) {
    split_finish_kernel<<<(a.M + kFinishWarps - 1) / kFinishWarps, 32 * kFinishWarps, 0, st>>>(a, far_chunks, b, vpart);
    return cudaGetLastError();
}

}  // namespace rf
