// lu.cu - the direct variant of the solve: dense LU factorisation with
// partial pivoting and the triangular solves, FP64 on the device.
//
// Reference: LAPACK dgesv called by fortran/coeffs_and_vels.f90:62,158,333,514
// (the *_direct golden runs).  Blocked right-looking factorisation of panels
// of kLuNb = 128 columns; right-hand sides stand as further columns behind the
// matrix and go through the same swaps, triangles and updates, so that the
// forward substitution needs no pass of its own:
//   lu_panel_kernel         one cluster factors W columns of the tall panel in
//                           its registers (pivot: first row of largest
//                           magnitude, as idamax);
//   lu_panel_update_kernel  the W columns' update of the rest of the panel,
//                           over the whole GPU;
//   lu_trsm_kernel          the panel's row swaps on the trailing columns and
//                           U12 = L11^-1 A12 in shared memory, block by block
//                           on the FP64 tensor cores;
//   lu_gemm_kernel          A22 -= L21 U12, the rank-128 trailing update on
//                           the FP64 tensor cores: most of the 2/3 n^3 flops;
//   lu_back_kernel          back substitution, 128 rows at a time.
// The swaps are not applied to the L columns left of a panel: nothing reads
// them again.  Info as LAPACK: the first zero pivot (1-based), 0 when there
// is none.
//
// What bounds it (n = 15000): the trailing updates, 78 of 122 ms = 29 of 37
// TFLOP/s (128-column panels: the 64-column panels of a cuBLAS GEMM before
// passed twice as often over the trailing matrix, 107 ms), then the panels, 31
// ms: 1.4 us a column, three quarters of it latencies of the pivot search, the
// exchange and the cluster barrier.  Before, a panel went through memory eight
// columns at a time (92 ms, and 36 ms of rank-8 updates), the triangles ran one
// thread per column through global memory and the forward substitution panel
// by panel.  Factor and solve: n = 15000 234 -> 122 ms, n = 4500 37 -> 13 ms,
// n = 1500 10.7 -> 3.4 ms, n = 300 2.0 -> 0.7 ms; rf_dgesv n = 3001 with its
// copies 34 -> 17 ms.
#include <cooperative_groups.h>

#include <algorithm>

#include "rf_kernels.h"

namespace rf {
namespace {

namespace cg = cooperative_groups;

constexpr int kLuNb = 128;
constexpr int kPanelThreads = 256;
constexpr int kPanelWarps = kPanelThreads / 32;
constexpr int kMaxCluster = 16;
constexpr unsigned kNoRow = 0xffffffffu;
constexpr double kMinNormal = 2.2250738585072014e-308, kSubScale = 18446744073709551616.0;  // 2^-1022, 2^64

// A pivot candidate: |value| as an ordered integer (high and low word; none and
// NaN: 0 with row kNoRow, but a NaN on the diagonal stands as a zero, so that a
// column of NaN keeps its row) and its row index; then a row of values.
struct alignas(16) Pivot {
    unsigned hi, lo, row, pad;
};
template <int W>
struct PanelSlot {
    Pivot p;
    double v[W + W % 2];
};

// The first maximum over a warp, to every lane; returns the lane that had it.
// Usually one lane has the largest high word; otherwise the low words and then
// the row indices decide.
__device__ __forceinline__ int warp_first_max(Pivot &p) {
    const unsigned h = __reduce_max_sync(0xffffffffu, p.hi);
    unsigned b = __ballot_sync(0xffffffffu, p.hi == h);
    if (__popc(b) != 1) {
        const unsigned l = __reduce_max_sync(0xffffffffu, p.hi == h ? p.lo : 0u);
        const bool at = p.hi == h && p.lo == l;
        const unsigned r = __reduce_min_sync(0xffffffffu, at ? p.row : kNoRow);
        b = __ballot_sync(0xffffffffu, at && p.row == r);
    }
    const int src = __ffs(b) - 1;
    p.hi = h;
    p.lo = __shfl_sync(0xffffffffu, p.lo, src);
    p.row = __shfl_sync(0xffffffffu, p.row, src);
    return src;
}

// a row of W values between registers and (16-byte aligned) shared memory
template <int W>
__device__ __forceinline__ void store_row(double *s, const double (&v)[W]) {
#pragma unroll
    for (int e = 0; e + 1 < W; e += 2) *reinterpret_cast<double2 *>(s + e) = make_double2(v[e], v[e + 1]);
    if (W % 2) s[W - 1] = v[W - 1];
}
template <int W>
__device__ __forceinline__ void load_row(double (&v)[W], const double *s) {
#pragma unroll
    for (int e = 0; e + 1 < W; e += 2) {
        const double2 t = *reinterpret_cast<const double2 *>(s + e);
        v[e] = t.x;
        v[e + 1] = t.y;
    }
    if (W % 2) v[W - 1] = s[W - 1];
}

// far from both ends of the range, 2^-959 <= |v| < 2^960 (and so not zero,
// infinite or NaN): rcp_pos holds its bound and div_by's products and remainder
// are normal numbers.  On the exponent: two integer operations, where FP64
// comparisons stood in the serial chain of the back substitution.
__device__ __forceinline__ bool mid_range(double v) {
    constexpr unsigned lo = 64u << 20, hi = 1983u << 20;
    return ((unsigned)__double2hiint(v) & 0x7fffffffu) - lo < hi - lo;
}

// The interchanges of slots 0..w-1 with slots to[0..w-1] (to[t] >= t; slot
// W + t is a row below the triangle that turn t names first) in turn, as one
// permutation: src[s] = the slot whose row ends in slot s.  Not by stepping
// through them: what stands in slot t when its turn comes is what stood in slot
// par(t), the last earlier turn that named t, when that turn came, and so on
// back to a slot nobody named (root); slot t ends with what stood in slot to[t]
// at that moment, which the last earlier turn with the same target put there.
// last: per group of 32 turns the last one that names each slot; par and last
// are scratch.  Needs w <= 32 G threads; barriers inside and around it.
template <int G, int W>
__device__ __forceinline__ void swaps_to_permutation(const int *to, int w, int *par, int (*last)[2 * W], int *src) {
    const int t = threadIdx.x, grp = t >> 5;
    for (int e = t; e < G * 2 * W; e += blockDim.x) last[e / (2 * W)][e % (2 * W)] = -1;
    if (t < W) par[t] = t;
    __syncthreads();
    const int mine = t < w ? to[t] : -1 - t;
    unsigned same = 0;
    if (t < 32 * G) {
        same = __match_any_sync(0xffffffffu, mine);
        if (t < w && (same >> (t & 31)) == 1u) last[grp][mine] = t;  // the last of its group
    }
    __syncthreads();
    // every other turn that names slot t comes before t
    if (t < W) {
        int q = -1;
        for (int e = 0; e < G; ++e)
            if (last[e][t] != t) q = max(q, last[e][t]);
        const unsigned below = t < w && mine == t ? same & ((1u << (t & 31)) - 1u) : 0u;  // its own group, itself left out
        if (below) q = max(q, (t & ~31) + 31 - __clz(below));
        par[t] = q >= 0 ? q : t;
    }
    __syncthreads();
    auto root = [&](int r) {
        while (par[r] != r) r = par[r];
        return r;
    };
    if (t < w) {
        const unsigned below = same & ((1u << (t & 31)) - 1u);
        int before = below ? (t & ~31) + 31 - __clz(below) : -1;
        bool after = (same >> (t & 31)) != 1u;
        for (int e = 0; e < G; ++e) {
            if (e < grp && !below) before = max(before, last[e][mine]);
            if (e > grp && last[e][mine] >= 0) after = true;
        }
        src[t] = mine == t ? root(t) : before >= 0 ? root(before) : mine;
        if (mine >= W && !after) src[mine] = root(t);
        if (mine != W + t) src[W + t] = W + t;  // a slot without a row
    } else if (t < W) {
        src[t] = t;
        src[W + t] = W + t;
    }
}

// Sub-panel factorisation: columns [s0, s0 + w), w <= W, of the panel [k, k +
// nb) on one cluster, up to R rows per thread (row s0 + g + u x cluster threads
// for thread g), at most 64 values each, in registers.  A step is the pivot
// search (integer reductions over a warp, then over the CTA's candidates), one
// exchange in which every CTA writes its candidate to a slot in the shared
// memory of every CTA of the cluster, one cluster barrier, and the swap,
// scaling and rank-1 update; no global memory.  The row of the diagonal
// belongs to thread j of the first CTA, which sends it along.  Slots alternate
// between two buffers: a CTA that writes step j + 2's candidate has passed
// step j + 1's barrier, which every CTA reaches only after it has read step j's.
// A step always works on value 0 of a row and rotates the row by one place
// (the update writes value c to place c - 1), so that the steps are one loop:
// unrolled, each step's code ran once and cold, 3.7 us a column instead of 1.4.
// The finished columns ride along at the end of the row, updated with a
// multiplier row of zeros and swapped like the rest.  Then the sub-panel is
// written back and the cluster's CTAs take the panel's other columns in turn:
// the w swaps as one permutation of the at most 2w rows they touch, and for
// columns on the right U (unit lower w x w triangle).
template <int R, int W>
__global__ void __launch_bounds__(kPanelThreads) lu_panel_kernel(double *A, int64_t lda, int64_t n, int64_t k, int nb,
                                                                 int64_t s0, int w, int *piv, int *info) {
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = cluster.block_rank(), ranks = cluster.num_blocks();
    __shared__ PanelSlot<W> s_cand[2][kMaxCluster];  // every CTA's candidate, the finished columns' values zero
    __shared__ Pivot s_warp[kPanelWarps];
    constexpr int WA = W + W % 2;                    // rows start on 16 bytes
    __shared__ __align__(16) double s_win[WA];       // the CTA's candidate's row before it is sent
    __shared__ __align__(16) double s_own[WA];       // first CTA: the diagonal's, likewise
    __shared__ __align__(16) double s_diag[2][WA];   // the diagonal's row
    __shared__ __align__(16) double s_full[2][kMaxCluster][WA];  // first CTA: the candidates' whole rows
    __shared__ long long s_row[2 * W];               // rows of the permutation's slots
    __shared__ int s_src[2 * W], s_last[1][2 * W];
    __shared__ int s_to[W], s_par[W];
    __shared__ unsigned s_piv[W];
    __shared__ double s_l[W][W + 1];
    __shared__ double s_v[kPanelWarps][2 * W];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t g = (int64_t)rank * kPanelThreads + tid, stride = (int64_t)ranks * kPanelThreads;
    double v[R][W];
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int64_t r = s0 + g + u * stride;
#pragma unroll
        for (int c = 0; c < W; ++c) v[u][c] = r < n && c < w ? A[(s0 + c) * lda + r] : 0.0;
    }
#pragma unroll 1
    for (int j = 0; j < w; ++j) {
        const int64_t col = s0 + j;
        const int buf = j & 1;
        // this thread's first maximum, the warp's, the CTA's
        Pivot mine{0, 0, g == j ? (unsigned)col : kNoRow, 0};
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int64_t r = s0 + g + u * stride;
            const double x = fabs(v[u][0]);
            if (r >= col && r < n && x == x) {
                const unsigned xh = __double2hiint(x), xl = __double2loint(x);
                if (mine.row == kNoRow || xh > mine.hi || (xh == mine.hi && xl > mine.lo))
                    mine.hi = xh, mine.lo = xl, mine.row = (unsigned)r;
            }
        }
        Pivot c = mine;
        if (lane == warp_first_max(c)) s_warp[warp] = c;
        __syncthreads();
        c = lane < kPanelWarps ? s_warp[lane] : Pivot{0, 0, kNoRow, 0};
        warp_first_max(c);
        if (mine.row == c.row && c.row != kNoRow) {  // the owner
#pragma unroll
            for (int u = 0; u < R; ++u)
                if (s0 + g + u * stride == (int64_t)c.row) store_row<W>(s_win, v[u]);
        }
        if (g == j) store_row<W>(s_own, v[0]);
        __syncthreads();
        // the CTA's candidate (first CTA: and the diagonal's row) to every CTA
        {
            const double x = lane < W ? s_win[lane] : 0.0, y = lane < W ? s_own[lane] : 0.0;
            for (int q = warp; q < ranks; q += kPanelWarps) {
                PanelSlot<W> *dst = cluster.map_shared_rank(&s_cand[buf][rank], q);
                if (lane == 0) dst->p = c;
                if (lane < W) {
                    dst->v[lane] = lane < w - j ? x : 0.0;
                    if (q == 0) cluster.map_shared_rank(s_full[buf][rank], 0)[lane] = x;
                    if (rank == 0) cluster.map_shared_rank(s_diag[buf], q)[lane] = y;
                }
            }
        }
        cluster.sync();
        // the cluster's first maximum
        c = lane < ranks ? s_cand[buf][lane].p : Pivot{0, 0, kNoRow, 0};
        const int slot = warp_first_max(c) % ranks;
        const PanelSlot<W> &win = s_cand[buf][slot];
        const int64_t p = c.row;
        const double d = win.v[0];
        if (tid == 0) s_piv[j] = c.row;
        if (rank == 0 && tid == 0) {
            piv[col] = (int)c.row;
            if (d == 0.0 && *info == 0) *info = (int)(col + 1);
        }
        double inv = div_by(1.0, d, copysign(rcp_pos(fabs(d)), d));  // 1/d as the division gives it, where d is in mid range
        if (p != col) {
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const int64_t r = s0 + g + u * stride;
                if (r == p) load_row<W>(v[u], s_diag[buf]);
                else if (r == col) load_row<W>(v[u], s_full[buf][slot]);  // the first CTA's
            }
        }
        if (!mid_range(d)) {
            // a zero pivot leaves its column (dgetf2).  A subnormal one's reciprocal
            // overflows: pivot and column are scaled up, which is exact (no entry
            // is larger than the pivot); dgetf2 divides there.
            const double up = fabs(d) < kMinNormal ? kSubScale : 1.0;
            inv = d != 0.0 ? 1.0 / (d * up) : 1.0;
#pragma unroll
            for (int u = 0; u < R; ++u)
                if (s0 + g + u * stride > col) v[u][0] *= up;
        }
        double nx[R];  // minus the multiplier; rows above keep their values
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const bool below = s0 + g + u * stride > col;
            if (below) v[u][0] *= inv;
            nx[u] = below ? -v[u][0] : 0.0;
        }
        double first[R];
#pragma unroll
        for (int u = 0; u < R; ++u) first[u] = v[u][0];
#pragma unroll
        for (int c = 1; c < W; ++c) {
            const double m = win.v[c];
#pragma unroll
            for (int u = 0; u < R; ++u) v[u][c - 1] = fma(nx[u], m, v[u][c]);
        }
#pragma unroll
        for (int u = 0; u < R; ++u) v[u][W - 1] = first[u];
    }
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const int64_t r = s0 + g + u * stride;
        if (r < n) {
#pragma unroll
            for (int c = 0; c < W; ++c) {
                const int cc = (c + w) % W;  // place c holds column c + w, rotated
                if (cc < w) A[(s0 + cc) * lda + r] = v[u][c];
            }
        }
    }
    __threadfence();
    cluster.sync();  // the w x w triangle, written by the first CTA, is read by all
    for (int t = tid; t < w * w; t += kPanelThreads) s_l[t % w][t / w] = __ldcg(&A[(s0 + t / w) * lda + s0 + t % w]);
    // slot t < W is row s0 + t, slot W + t is pivot row t where it lies below
    // the triangle and was not named before
    if (tid < 32) {
        const unsigned p = tid < w ? s_piv[tid] : kNoRow - 1 - tid;
        const int firstp = __ffs(__match_any_sync(0xffffffffu, p)) - 1;
        if (tid < W) {
            const bool below = tid < w && (int64_t)p >= s0 + w;
            s_to[tid] = tid >= w ? tid : below ? W + firstp : (int)((int64_t)p - s0);
            s_row[tid] = tid < w ? (long long)(s0 + tid) : -1LL;
            s_row[W + tid] = below && firstp == tid ? (long long)p : -1LL;
        }
    }
    __syncthreads();
    swaps_to_permutation<1, W>(s_to, w, s_par, s_last, s_src);
    __syncthreads();
    // a column per warp
    for (int64_t c0 = k + (int64_t)rank * kPanelWarps; c0 < k + nb; c0 += (int64_t)ranks * kPanelWarps) {
        auto other = [&](int64_t c) { return c < k + nb && (c < s0 || c >= s0 + w); };
#pragma unroll 2
        for (int e = tid; e < kPanelWarps * 2 * W; e += kPanelThreads) {
            const int sl = e % (2 * W);
            const int64_t c = c0 + e / (2 * W);
            if (other(c) && s_row[sl] >= 0) s_v[e / (2 * W)][sl] = A[c * lda + s_row[s_src[sl]]];
        }
        __syncthreads();
        if (c0 + warp >= s0 + w) {  // right of the sub-panel: U, x_i -= l_iq x_q, q in turn
            double x = lane < w ? s_v[warp][lane] : 0.0;
            for (int q = 0; q + 1 < w; ++q) {
                const double xq = __shfl_sync(0xffffffffu, x, q);
                if (lane > q && lane < w) x = fma(-s_l[lane][q], xq, x);
            }
            if (lane < w) s_v[warp][lane] = x;
        }
        __syncthreads();
#pragma unroll 2
        for (int e = tid; e < kPanelWarps * 2 * W; e += kPanelThreads) {
            const int sl = e % (2 * W);
            const int64_t c = c0 + e / (2 * W);
            if (other(c) && s_row[sl] >= 0) A[c * lda + s_row[sl]] = s_v[e / (2 * W)][sl];
        }
        __syncthreads();
    }
}

// The sub-panel's rank-w update of the panel's columns right of it:
// A[r, c] -= sum_q A[r, s0 + q] A[s0 + q, c] for rows r >= s0 + w and columns c
// in [s0 + w, k + nb); one thread per row and group of kUpdCols columns
// (blockIdx.y), the U entries in shared memory.
constexpr int kUpdCols = 8;
constexpr int kUpdThreads = 128;
template <int W>
__global__ void __launch_bounds__(kUpdThreads) lu_panel_update_kernel(double *A, int64_t lda, int64_t n, int64_t k,
                                                                      int nb, int64_t s0, int w) {
    __shared__ double s_uu[kUpdCols][W];
    const int64_t c0 = s0 + w + (int64_t)blockIdx.y * kUpdCols;
    const int nc = (int)std::min<int64_t>(k + nb - c0, kUpdCols);
    for (int t = threadIdx.x; t < kUpdCols * W; t += kUpdThreads) {
        const int c = t / W, q = t % W;
        s_uu[c][q] = c < nc && q < w ? A[(c0 + c) * lda + s0 + q] : 0.0;
    }
    __syncthreads();
    const int64_t r = s0 + w + blockIdx.x * (int64_t)kUpdThreads + threadIdx.x;
    if (r >= n) return;
    double l[W], v[kUpdCols];
#pragma unroll
    for (int q = 0; q < W; ++q) l[q] = q < w ? A[(s0 + q) * lda + r] : 0.0;
#pragma unroll
    for (int c = 0; c < kUpdCols; ++c) v[c] = c < nc ? A[(c0 + c) * lda + r] : 0.0;
#pragma unroll
    for (int c = 0; c < kUpdCols; ++c) {
#pragma unroll
        for (int q = 0; q < W; ++q) v[c] = fma(-l[q], s_uu[c][q], v[c]);
        if (c < nc) A[(c0 + c) * lda + r] = v[c];
    }
}

// The panel's swaps on the trailing columns [k + nb, ncols), then U12 = L11^-1
// A12 (L11 unit lower, nb x nb).  A CTA owns kTrsmCols columns.  The swaps are
// one permutation of the at most 2 nb rows they touch: the panel's rows come
// into shared memory through it (a thread per row, lanes along the rows), and a
// pivot row below the panel, which can only receive a row of the panel, takes
// it straight from the column.  The triangle goes by blocks of 32 rows: a
// block's earlier rows are taken off on the FP64 tensor cores (a warp per eight
// columns; with fused multiply-adds from shared memory these 32 x 32 steps
// were bound by its bandwidth, 51 of 120 thousand cycles), then one thread per
// column solves the block's own triangle in registers.
constexpr int kTrsmB = 32;
constexpr int kTrsmCols = 64;
constexpr int kTrsmThreads = 256;
constexpr int kTrsmLd = kTrsmCols + 4;  // 4 mod 16 doubles, as kTrsmLdL
constexpr int kTrsmLdL = kTrsmB + 4;
__global__ void __launch_bounds__(kTrsmThreads) lu_trsm_kernel(double *A, int64_t lda, int64_t ncols, int64_t k, int nb,
                                                               const int *piv) {
    __shared__ __align__(16) double s_l[kTrsmB][kTrsmLdL];  // [column][row] of the current block of L11
    __shared__ int64_t s_row[2 * kLuNb];
    __shared__ int s_src[2 * kLuNb], s_last[kLuNb / 32][2 * kLuNb];
    __shared__ int s_to[kLuNb], s_par[kLuNb], s_piv[kLuNb];
    extern __shared__ double s_x[];  // [nb][kTrsmLd]: the panel's rows of every column
    const int tid = threadIdx.x;
    if (tid < kLuNb) s_piv[tid] = tid < nb ? piv[k + tid] : -1;
    __syncthreads();
    if (tid < kLuNb) {
        const int p = s_piv[tid];
        int first = tid;
#pragma unroll 16
        for (int q = kLuNb - 1; q >= 0; --q)
            if (q < tid && s_piv[q] == p) first = q;
        const bool below = tid < nb && p >= k + nb;
        s_to[tid] = tid >= nb ? tid : below ? kLuNb + first : (int)(p - k);
        s_row[tid] = k + tid;
        s_row[kLuNb + tid] = below && first == tid ? p : -1;
    }
    __syncthreads();
    swaps_to_permutation<kLuNb / 32, kLuNb>(s_to, nb, s_par, s_last, s_src);
    __syncthreads();
    const int64_t c0 = k + nb + blockIdx.x * (int64_t)kTrsmCols;
    const int nc = (int)std::min<int64_t>(kTrsmCols, ncols - c0);
    // thread: row t of the panel, columns ch, ch + 2, ...
    static_assert(kTrsmThreads == 2 * kLuNb, "a thread per row and half the columns");
    const int t = tid % kLuNb, ch = tid / kLuNb;
    {
        const double *from = A + c0 * lda + s_row[s_src[t < nb ? t : 0]];
#pragma unroll 16
        for (int c = ch; c < kTrsmCols; c += 2) s_x[t * kTrsmLd + c] = t < nb && c < nc ? from[c * lda] : 0.0;
    }
    __syncthreads();
    // the displaced rows; the panel's own rows are still as they were in A
    if (t < nb && s_row[kLuNb + t] >= 0) {
        const double *from = A + c0 * lda + s_row[s_src[kLuNb + t]];
        double *to = A + c0 * lda + s_row[kLuNb + t];
        for (int cb = ch; cb < nc; cb += 16) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = cb + 2 * u < nc ? from[(cb + 2 * u) * lda] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (cb + 2 * u < nc) to[(cb + 2 * u) * lda] = v[u];
        }
    }
    const int lane = tid & 31, wc = 8 * (tid >> 5), g = lane >> 2, q4 = lane & 3;
    // the next block of L11 is on its way while one is used
    constexpr int kPer = kTrsmB * kTrsmB / kTrsmThreads;
    double next[kPer];
    auto fetch = [&](int b, int q0) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int e = tid + u * kTrsmThreads, i = e % kTrsmB, q = e / kTrsmB;
            next[u] = b + i < nb && q0 + q < nb ? A[(k + q0 + q) * lda + k + b + i] : 0.0;
        }
    };
    fetch(0, 0);
    for (int b = 0; b < nb; b += kTrsmB) {
        double d[4][2];  // minus the block: rows 8 i + g, columns wc + 2 q4 + {0, 1}
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) d[i][h] = 0.0;
        for (int q0 = 0; q0 <= b; q0 += kTrsmB) {
            __syncthreads();  // s_x is loaded, the block before has been used
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                const int e = tid + u * kTrsmThreads;
                s_l[e / kTrsmB][e % kTrsmB] = next[u];
            }
            if (q0 < b) fetch(b, q0 + kTrsmB);
            else fetch(b + kTrsmB, 0);
            __syncthreads();
            if (q0 < b) {
#pragma unroll
                for (int q = 0; q < kTrsmB; q += 4) {
                    const double x = s_x[(q0 + q + q4) * kTrsmLd + wc + g];
#pragma unroll
                    for (int i = 0; i < 4; ++i) dmma_8x8x4(d[i][0], d[i][1], s_l[q + q4][8 * i + g], x, d[i][0], d[i][1]);
                }
            }
        }
        // the block's rows less the earlier rows' part, then its triangle
        if (b > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) s_x[(b + 8 * i + g) * kTrsmLd + wc + 2 * q4 + h] -= d[i][h];
            __syncthreads();
        }
        if (tid < kTrsmCols) {
            double x[kTrsmB];
#pragma unroll
            for (int i = 0; i < kTrsmB; ++i) x[i] = s_x[(b + i) * kTrsmLd + tid];
#pragma unroll
            for (int q = 0; q < kTrsmB; ++q)
#pragma unroll
                for (int i = q + 1; i < kTrsmB; ++i) x[i] = fma(-s_l[q][i], x[q], x[i]);
#pragma unroll
            for (int i = 0; i < kTrsmB; ++i) s_x[(b + i) * kTrsmLd + tid] = x[i];
        }
    }
    __syncthreads();
    if (t < nb) {
        double *to = A + c0 * lda + k + t;
#pragma unroll 16
        for (int c = ch; c < kTrsmCols; c += 2)
            if (c < nc) to[c * lda] = s_x[t * kTrsmLd + c];
    }
}

// C -= A B on the FP64 tensor cores (mma.sync m8n8k4): A m x kLuNb, B kLuNb x
// nc, C m x nc, all column-major with ld lda and 16-byte aligned starts.  A CTA
// of four warps owns a 128 x 64 tile, a warp 64 x 32 of it in registers;
// operands in k-blocks of 16 through a ring of three stages (cp.async).  The
// products are summed by themselves and C taken off behind the second half of
// the k-blocks, a thread's rows in turn (on average 28 of 128 products are
// added to sums that hold C).  Summed onto C from the start, every product was
// rounded at C's size: error of a solution at n = 2500 2.8e-15, from zero with C
// loaded at the end 0.8e-15 but 174 instead of 126 ms at n = 15000; this way
// 1.5e-15 (LAPACK's 1.4e-15) and 122 ms, C's loads now behind the products.  Two
// CTAs per SM: one's C traffic hides behind the other's products.  Row strides
// of 4 mod 16 doubles keep the operand loads free of bank conflicts.
constexpr int kGM = 128, kGN = 64, kGK = 16, kGStages = 3, kGThreads = 128;
constexpr int kGLdA = kGM + 4, kGLdB = kGK + 4;
constexpr size_t kGStage = sizeof(double) * (kGK * kGLdA + kGN * kGLdB);

__device__ __forceinline__ void cp16(void *dst, const void *src, int bytes) {  // the rest of the 16 bytes is zero
    const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(LEFT) : "memory");
}

__global__ void __launch_bounds__(kGThreads, 2) lu_gemm_kernel(const double *__restrict__ A,
                                                               const double *__restrict__ B, double *__restrict__ C,
                                                               int64_t lda, int64_t m, int64_t nc) {
    extern __shared__ __align__(16) double smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t r0 = (int64_t)blockIdx.x * kGM, c0 = (int64_t)blockIdx.y * kGN;
    // within the tile 32-bit offsets do (128 columns of less than 2^24 rows)
    A += r0;
    B += c0 * lda;
    C += c0 * lda + r0;
    const int ld = (int)lda, rows = (int)std::min<int64_t>(m - r0, kGM), cols = (int)std::min<int64_t>(nc - c0, kGN);
    auto stage_a = [&](int st) { return smem + st * (kGK * kGLdA + kGN * kGLdB); };
    auto stage_b = [&](int st) { return stage_a(st) + kGK * kGLdA; };
    auto load = [&](int kb) {
        double *sa = stage_a(kb % kGStages), *sb = stage_b(kb % kGStages);
        const int k0 = kb * kGK;
#pragma unroll
        for (int t = 0; t < kGK * kGM / 2 / kGThreads; ++t) {
            const int e = t * kGThreads + tid, q = e / (kGM / 2), r = 2 * (e % (kGM / 2));
            cp16(sa + q * kGLdA + r, A + (k0 + q) * ld + (r < rows ? r : 0), r + 1 < rows ? 16 : r < rows ? 8 : 0);
        }
#pragma unroll
        for (int t = 0; t < kGN * kGK / 2 / kGThreads; ++t) {
            const int e = t * kGThreads + tid, c = e / (kGK / 2), q = 2 * (e % (kGK / 2));
            cp16(sb + c * kGLdB + q, B + (c < cols ? c : 0) * ld + k0 + q, c < cols ? 16 : 0);
        }
    };
    constexpr int KB = kLuNb / kGK;
#pragma unroll
    for (int s = 0; s < kGStages - 1; ++s) {
        load(s);
        cp_commit();
    }
    const int wr = (warp & 1) * 64, wc = (warp >> 1) * 32;
    const int g = lane >> 2, q4 = lane & 3;
    double acc[8][4][2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    auto arrive = [&](int kb) {
        cp_wait<kGStages - 2>();
        __syncthreads();  // stage kb has arrived for every thread, stage kb - 1 has been read
        if (kb + kGStages - 1 < KB) load(kb + kGStages - 1);
        cp_commit();
    };
    auto products = [&](int kb, int s0, int s1) {
        const double *sa = stage_a(kb % kGStages) + q4 * kGLdA + wr + g;
        const double *sb = stage_b(kb % kGStages) + (wc + g) * kGLdB + q4;
#pragma unroll
        for (int s = s0; s < s1; s += 4) {
            double a[8], b[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = sa[s * kGLdA + 8 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = sb[8 * j * kGLdB + s];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j], acc[i][j][0], acc[i][j][1]);
        }
    };
#pragma unroll 1
    for (int kb = 0; kb < KB / 2; ++kb) {
        arrive(kb);
        products(kb, 0, kGK);
    }
    // C comes in behind the second half, the values of one of a thread's rows at a
    // time (addresses clamped to the tile, not predicated: branches here took 57
    // doubles of local memory)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int kb = KB / 2 + i / 2;
        double old[4][2];
        const int r = min(wr + 8 * i + g, rows - 1);  // beyond the tile: never stored
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) old[j][h] = C[min(wc + 8 * j + 2 * q4 + h, cols - 1) * ld + r];
        if (i % 2 == 0) arrive(kb);
        products(kb, i % 2 * (kGK / 2), (i % 2 + 1) * (kGK / 2));
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) acc[i][j][h] -= old[j][h];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int c = wc + 8 * j + 2 * q4 + h;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int r = wr + 8 * i + g;
                if (r < rows && c < cols) C[c * ld + r] = -acc[i][j][h];
            }
        }
}

// Back substitution, rows [k, k + nb): the triangle in shared memory, by blocks
// of 32 rows from the last (one warp, the block's rows in its lanes, x_p
// broadcast by shuffles), each solved block taken off the rows above it by all
// warps.  Quotients come from each lane's reciprocal; a block in which a pivot,
// an operand or a quotient is zero, not finite or near the ends of the range is
// solved again with divisions (a subnormal or huge pivot has no usable
// reciprocal; overflow and underflow need the division's own rounding).  A
// choice per quotient stood in the serial chain: 20.5 instead of 15.1 us a block.
constexpr int kBackThreads = 512;
constexpr int kBackLd = kLuNb + 1;
__global__ void __launch_bounds__(kBackThreads) lu_back_diag_kernel(const double *__restrict__ A, int64_t lda,
                                                                    int64_t k, int nb, double *x) {
    extern __shared__ double s_u[];  // [column][kBackLd]
    __shared__ double s_x[kLuNb];
    __shared__ double s_p[4][kLuNb];
    const int tid = threadIdx.x, lane = tid & 31;
    for (int t = tid; t < nb; t += kBackThreads) s_x[t] = x[k + t];
#pragma unroll 16
    for (int t = tid; t < kLuNb * kLuNb; t += kBackThreads) {
        const int i = t % kLuNb, p = t / kLuNb;
        if (i <= p && p < nb) s_u[p * kBackLd + i] = A[(k + p) * lda + k + i];
    }
    __syncthreads();
    for (int b = (nb - 1) / 32 * 32; b >= 0; b -= 32) {
        const int bn = min(32, nb - b);
        if (tid < 32) {
            const double x0 = lane < bn ? s_x[b + lane] : 0.0, d = lane < bn ? s_u[(b + lane) * kBackLd + b + lane] : 1.0;
            const double rd = copysign(rcp_pos(fabs(d)), d);
            double num;  // what the lane's quotient was formed from
            auto solve = [&](auto quotient) {
                double xi = num = x0;
                for (int p = bn - 1; p >= 0; --p) {
                    const double u = lane < p ? s_u[(b + p) * kBackLd + b + lane] : 0.0;
                    const double q = quotient(xi);  // every lane's: no branch
                    if (lane == p) num = xi, xi = q;
                    const double xp = __shfl_sync(0xffffffffu, xi, p);
                    if (lane < p) xi = fma(-u, xp, xi);
                }
                return xi;
            };
            double xi = solve([&](double v) { return div_by(v, d, rd); });
            const bool ok = mid_range(d) && mid_range(num) && mid_range(xi);
            if (__any_sync(0xffffffffu, !ok && lane < bn)) xi = solve([&](double v) { return v / d; });
            if (lane < bn) s_x[b + lane] = xi;
        }
        __syncthreads();
        // rows above: four threads per row, eight columns each
        const int i = tid % kLuNb, q = tid / kLuNb;
        if (i < b) {
            double v = 0.0;
#pragma unroll
            for (int p = 0; p < 8; ++p)
                if (8 * q + p < bn) v = fma(s_u[(b + 8 * q + p) * kBackLd + i], s_x[b + 8 * q + p], v);
            s_p[q][i] = v;
        }
        __syncthreads();
        if (tid < b) s_x[tid] -= (s_p[0][tid] + s_p[1][tid]) + (s_p[2][tid] + s_p[3][tid]);
        __syncthreads();
    }
    for (int t = tid; t < nb; t += kBackThreads) x[k + t] = s_x[t];
}

// x[r] -= sum_p A[r, k + p] x[k + p] for rows r < k: a CTA takes 32 rows, eight
// threads per row each an eighth of the columns (interleaved), added in order.
__global__ void __launch_bounds__(256) lu_back_update_kernel(const double *__restrict__ A, int64_t lda, int64_t k,
                                                             int nb, double *x) {
    __shared__ double s_x[kLuNb];
    __shared__ double s_p[8][32];
    const int tid = threadIdx.x, part = tid >> 5, lane = tid & 31;
    for (int t = tid; t < nb; t += 256) s_x[t] = x[k + t];
    __syncthreads();
    const int64_t r = blockIdx.x * (int64_t)32 + lane;
    double s = 0.0;
    if (r < k) {
#pragma unroll 8
        for (int p = part; p < nb; p += 8) s = fma(A[(k + p) * lda + r], s_x[p], s);
    }
    s_p[part][lane] = s;
    __syncthreads();
    if (part == 0 && r < k) {
        double v = x[r];
#pragma unroll
        for (int q = 0; q < 8; ++q) v -= s_p[q][lane];
        x[r] = v;
    }
}

int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

// rows that the largest cluster holds at R per thread
constexpr int64_t reg_rows(int R) { return (int64_t)R * kMaxCluster * kPanelThreads; }

// One sub-panel of w <= W columns on one cluster that holds its rows at R per
// thread, then its update of the panel's other columns.  At least eight CTAs,
// which share the panel's other columns at the end.
template <int R, int W>
cudaError_t sub_panel(double *A, int64_t lda, int64_t n, int64_t k, int nb, int64_t s0, int w, int *piv, int *info,
                      cudaStream_t st, int64_t *launches) {
    const int ranks = (int64_t)R * 8 * kPanelThreads >= n - s0 ? 8 : kMaxCluster;
    auto kern = lu_panel_kernel<R, W>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ranks);
    cfg.blockDim = dim3(kPanelThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, A, lda, n, k, nb, s0, w, piv, info);
    ++*launches;
    const int64_t right = k + nb - s0 - w, below = n - s0 - w;
    if (e == cudaSuccess && right > 0 && below > 0) {
        lu_panel_update_kernel<W><<<dim3((unsigned)cdiv(below, kUpdThreads), (unsigned)cdiv(right, kUpdCols)),
                                    kUpdThreads, 0, st>>>(A, lda, n, k, nb, s0, w);
        ++*launches;
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace

cudaError_t lu_factor(double *A, int64_t lda, int64_t n, int64_t ncols, int *piv, int *info, cudaStream_t st,
                      int64_t *launches) {
    if (n > reg_rows(64) || lda % 2 != 0 || lda < n || ncols < n) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(info, 0, sizeof(int), st);
    const size_t trsm_smem = sizeof(double) * kLuNb * kTrsmLd, gemm_smem = kGStages * kGStage;
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(lu_trsm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)trsm_smem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(lu_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem);
    for (int64_t k = 0; k < n && e == cudaSuccess; k += kLuNb) {
        const int nb = (int)std::min<int64_t>(kLuNb, n - k);
        for (int s0 = 0; s0 < nb && e == cudaSuccess;) {
            // the widest sub-panel whose rows fit the cluster's registers
            const int64_t rows = n - k - s0;
            int w = 0;
            auto go = [&](auto sub, int W) {
                w = std::min(W, nb - s0);
                e = sub(A, lda, n, k, nb, k + s0, w, piv, info, st, launches);
            };
            if (rows <= reg_rows(1)) go(sub_panel<1, 32>, 32);
            else if (rows <= reg_rows(2)) go(sub_panel<2, 32>, 32);
            else if (rows <= reg_rows(4)) go(sub_panel<4, 16>, 16);
            else if (rows <= reg_rows(8)) go(sub_panel<8, 8>, 8);
            else if (rows <= reg_rows(16)) go(sub_panel<16, 4>, 4);
            else if (rows <= reg_rows(32)) go(sub_panel<32, 2>, 2);
            else go(sub_panel<64, 1>, 1);
            s0 += w;
        }
        const int64_t cols = ncols - k - nb, rows = n - k - nb;
        if (e != cudaSuccess || cols <= 0) continue;
        lu_trsm_kernel<<<(unsigned)cdiv(cols, kTrsmCols), kTrsmThreads, trsm_smem, st>>>(A, lda, ncols, k, nb, piv);
        ++*launches;
        if (rows > 0) {
            // rows > 0: the panel is whole, nb = kLuNb
            lu_gemm_kernel<<<dim3((unsigned)cdiv(rows, kGM), (unsigned)cdiv(cols, kGN)), kGThreads, gemm_smem, st>>>(
                A + k * lda + k + nb, A + (k + nb) * lda + k, A + (k + nb) * lda + k + nb, lda, rows, cols);
            ++*launches;
        }
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t lu_back(const double *A, int64_t lda, int64_t n, double *x, cudaStream_t st, int64_t *launches) {
    const size_t smem = sizeof(double) * kLuNb * kBackLd;
    cudaError_t e = cudaFuncSetAttribute(lu_back_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    for (int64_t k = (n - 1) / kLuNb * kLuNb; k >= 0 && e == cudaSuccess; k -= kLuNb) {
        const int nb = (int)std::min<int64_t>(kLuNb, n - k);
        lu_back_diag_kernel<<<1, kBackThreads, smem, st>>>(A, lda, k, nb, x);
        ++*launches;
        if (k > 0) {
            lu_back_update_kernel<<<(unsigned)cdiv(k, 32), 256, 0, st>>>(A, lda, k, nb, x);
            ++*launches;
        }
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace rf
