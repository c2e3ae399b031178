// precond.cu - neighbour-block preconditioners for the right-preconditioned GMRES.
//
// The 3N x 3N diagonal blocks of A are the identity (matrix_assembly.f90:
// 489-492), so plain block-Jacobi is no preconditioning at all, and no
// block-diagonal correction helps either: the lowest eigenvalues of A belong
// to modes localised on two or three close fibers (a pair coupled by a block
// C has eigenvalues 1 +- sigma(C); a block-diagonal P maps them to
// 1/(1 -+ sigma) and keeps their ratio), the highest to modes spread over
// tens of fibers in the dense core.  What does help is coupling a fiber to
// its nearest neighbours:
//
//   z_i = v_i + sum_{m < kp} B_{i,m} v_{j_m},   j_m = the m-th nearest neighbour
//
// with B_{i,m} the coupling blocks of the local inverse:
//
//   RF_PC_CLUSTER  B_{i,m} = [S_i^-1]_{0, m+1}, S_i = A restricted to fiber i
//                  and its kc nearest neighbours (the exact local-cluster
//                  inverse); one CTA per fiber factorises S_i^T in shared
//                  memory (FP32 LU with partial pivoting) and keeps the
//                  first block row.
//   RF_PC_LEARNED  B_{i,m} predicted by a small MLP from the geometry of the
//                  16 nearest neighbours expressed in a frame attached to
//                  fiber i, neighbour m listed first (one evaluation per
//                  pair).  Blocks transform as B(Q config) = Q B(config) Q^T
//                  under rotations Q, and neighbour m's orientation enters
//                  with a canonical sign (the block's odd-order columns
//                  change sign with it), so the network only learns the
//                  rotation- and sign-free part.
//
// The MLP (144 -> 256 -> 256 -> 225, ReLU) is trained by the trainer below
// with the FP32 kernels of mlp_train.cu (forward, backward, Adam).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "handle.h"
#include "mlp_train.h"

namespace rf {
namespace {

constexpr int kK = RF_MLP_K;          // neighbours in the features
constexpr int kPair = RF_MLP_PAIRS;   // neighbour blocks per fiber
constexpr int kIn = RF_MLP_IN;        // 144
constexpr int kHid = RF_MLP_HIDDEN;   // 256
constexpr int kOut = RF_MLP_OUT;      // 225
constexpr int kNb = 15;               // block size the MLP is built for (N = 5)

// ------------------------------------------------------------------ k-NN
// One warp per fiber: every lane keeps the K nearest of its sources j = lane,
// lane + 32, ... sorted in registers (unrolled compare-and-swap), then K rounds
// of a warp arg-min over the lane heads merge them.  Order: distance, then the
// lower source index (the order of a sequential scan with strict comparison).
constexpr int kKnnWarps = 4;
__global__ void __launch_bounds__(kKnnWarps * 32) knn_kernel(int M, const double *__restrict__ pos, int K,
                                                             int *__restrict__ knn) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * kKnnWarps + (threadIdx.x >> 5);
    if (i >= M) return;  // whole warp
    float bd[kK];
    int bi[kK];
#pragma unroll
    for (int r = 0; r < kK; ++r) {
        bd[r] = 3.4e38f;
        bi[r] = 0x7fffffff;
    }
    const double xi = pos[3 * i], yi = pos[3 * i + 1], zi = pos[3 * i + 2];
    for (int j = lane; j < M; j += 32) {
        if (j == i) continue;
        const float dx = (float)(__ldg(pos + 3 * j) - xi), dy = (float)(__ldg(pos + 3 * j + 1) - yi),
                    dz = (float)(__ldg(pos + 3 * j + 2) - zi);
        float d = dx * dx + dy * dy + dz * dz;
        if (!(d < bd[kK - 1])) continue;
        int jj = j;
#pragma unroll
        for (int r = 0; r < kK; ++r) {
            if (d < bd[r]) {  // this lane's sources arrive in increasing j: ties keep the earlier one
                const float td = bd[r];
                const int ti = bi[r];
                bd[r] = d;
                bi[r] = jj;
                d = td;
                jj = ti;
            }
        }
    }
    for (int r = 0; r < K; ++r) {
        // lexicographic arg-min of (distance, index) over the lane heads
        float md = bd[0];
        int mi = bi[0];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float od = __shfl_xor_sync(0xffffffffu, md, o);
            const int oi = __shfl_xor_sync(0xffffffffu, mi, o);
            if (od < md || (od == md && oi < mi)) {
                md = od;
                mi = oi;
            }
        }
        if (lane == 0) knn[(int64_t)i * K + r] = mi < M ? mi : -1;
        if (bi[0] == mi && bd[0] == md) {  // the winning lane pops its head
#pragma unroll
            for (int q = 0; q < kK - 1; ++q) {
                bd[q] = bd[q + 1];
                bi[q] = bi[q + 1];
            }
            bd[kK - 1] = 3.4e38f;
            bi[kK - 1] = 0x7fffffff;
        }
    }
}

// ------------------------------------------------------------------ cluster inverse rows
// S = A[C, C] with C = {i, knn_0, .., knn_{kc-1}}; solve S^T X = E (E = the
// first nb columns of the identity) by LU with partial pivoting in shared
// memory: X^T is the first block row of S^-1, and its column blocks 1..kp are
// the couplings B_{i,m} (out[i][m], row-major nb x nb; zero for m >= kp).
template <typename T>
__global__ void __launch_bounds__(256) cluster_rows_kernel(int M, int nb, const T *__restrict__ A, int64_t lda,
                                                           int64_t plane, const int *__restrict__ knn, int kstride,
                                                           int kc, int kp, float *__restrict__ out,
                                                           int *__restrict__ singular) {
    extern __shared__ float sm[];
    __shared__ int s_fib[32];
    __shared__ int s_piv;
    __shared__ float s_pval;
    const int i = blockIdx.x;
    const int s = (kc + 1) * nb;
    const int w = s + nb;       // augmented width
    const int ld = w + 1;
    const int tid = threadIdx.x, nt = blockDim.x;
    if (tid <= kc) s_fib[tid] = tid == 0 ? i : knn[(int64_t)i * kstride + tid - 1];
    __syncthreads();
    // gather S^T: sm[r][c] = S[c][r] = A(row of cluster index c, column of r);
    // consecutive threads read consecutive rows of one column of A
    for (int idx = tid; idx < s * s; idx += nt) {
        const int r = idx / s, c = idx - r * s;
        const int64_t gr = (int64_t)s_fib[c / nb] * nb + c % nb;
        const int64_t gc = (int64_t)s_fib[r / nb] * nb + r % nb;
        sm[r * ld + c] = (float)load_entry<T>(A, gc * lda + gr, plane);
    }
    for (int idx = tid; idx < s * nb; idx += nt) {
        const int r = idx / nb, j = idx - r * nb;
        sm[r * ld + s + j] = (r == j) ? 1.f : 0.f;
    }
    __syncthreads();
    bool bad = false;
    for (int k = 0; k < s; ++k) {
        // pivot: warp 0 finds the largest |S[r][k]|, r >= k
        if (tid < 32) {
            float best = -1.f;
            int br = k;
            for (int r = k + tid; r < s; r += 32) {
                const float v = fabsf(sm[r * ld + k]);
                if (v > best) {
                    best = v;
                    br = r;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const float ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int orow = __shfl_xor_sync(0xffffffffu, br, o);
                if (ob > best || (ob == best && orow < br)) {
                    best = ob;
                    br = orow;
                }
            }
            if (tid == 0) {
                s_piv = br;
                s_pval = best;
            }
        }
        __syncthreads();
        if (!(s_pval > 0.f)) {
            bad = true;
            break;
        }
        const int p = s_piv;
        if (p != k)
            for (int c = k + tid; c < w; c += nt) {
                const float t = sm[k * ld + c];
                sm[k * ld + c] = sm[p * ld + c];
                sm[p * ld + c] = t;
            }
        __syncthreads();
        const float inv = 1.f / sm[k * ld + k];
        for (int r = k + 1 + tid; r < s; r += nt) sm[r * ld + k] *= inv;
        __syncthreads();
        const int rows = s - k - 1, cols = w - k - 1;
        for (int idx = tid; idx < rows * cols; idx += nt) {
            const int rr = idx / cols, cc = idx - rr * cols;
            const int r = k + 1 + rr, c = k + 1 + cc;
            sm[r * ld + c] -= sm[r * ld + k] * sm[k * ld + c];
        }
        __syncthreads();
    }
    float *dst = out + (int64_t)i * kPair * nb * nb;
    if (bad) {
        if (tid == 0) atomicAdd(singular, 1);
        for (int idx = tid; idx < kPair * nb * nb; idx += nt) dst[idx] = 0.f;  // P = I for this fiber
        return;
    }
    // back substitution on the nb right-hand sides, column-oriented: x_k,
    // then remove its contribution from the rows above
    for (int k = s - 1; k >= 0; --k) {
        if (tid < nb) sm[k * ld + s + tid] /= sm[k * ld + k];
        __syncthreads();
        for (int idx = tid; idx < k * nb; idx += nt) {
            const int r = idx / nb, j = idx - r * nb;
            sm[r * ld + s + j] -= sm[r * ld + k] * sm[k * ld + s + j];
        }
        __syncthreads();
    }
    // B_{i,m}[a][b] = (S^-1)[a][(m+1) nb + b] = X[(m+1) nb + b][a]
    for (int idx = tid; idx < kPair * nb * nb; idx += nt) {
        const int m = idx / (nb * nb), e = idx - m * nb * nb;
        const int a = e / nb, b = e - a * nb;
        dst[idx] = m < kp ? sm[((m + 1) * nb + b) * ld + s + a] : 0.f;
    }
}

// ------------------------------------------------------------------ features
// Frame of fiber i: e3 = t_i, e1 = the direction to the nearest neighbour
// with its t_i component removed, e2 = e3 x e1 (rows of E).
__device__ void fiber_frame(const double *__restrict__ pos, const double *__restrict__ ori, int i, int j0,
                            double E[3][3]) {
    const double *xi = pos + 3 * i, *ti = ori + 3 * i;
    const double e3[3] = {ti[0], ti[1], ti[2]};
    const double d1[3] = {pos[3 * j0] - xi[0], pos[3 * j0 + 1] - xi[1], pos[3 * j0 + 2] - xi[2]};
    double dot = d1[0] * e3[0] + d1[1] * e3[1] + d1[2] * e3[2];
    double e1[3] = {d1[0] - dot * e3[0], d1[1] - dot * e3[1], d1[2] - dot * e3[2]};
    double n1 = sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    if (n1 < 1e-9) {  // neighbour on the axis: any perpendicular direction
        const double a[3] = {fabs(e3[0]) < 0.9 ? 1.0 : 0.0, fabs(e3[0]) < 0.9 ? 0.0 : 1.0, 0.0};
        dot = a[0] * e3[0] + a[1] * e3[1];
        e1[0] = a[0] - dot * e3[0];
        e1[1] = a[1] - dot * e3[1];
        e1[2] = -dot * e3[2];
        n1 = sqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    }
    for (int a = 0; a < 3; ++a) e1[a] /= n1;
    const double e2[3] = {e3[1] * e1[2] - e3[2] * e1[1], e3[2] * e1[0] - e3[0] * e1[2], e3[0] * e1[1] - e3[1] * e1[0]};
    for (int c = 0; c < 3; ++c) {
        E[0][c] = e1[c];
        E[1][c] = e2[c];
        E[2][c] = e3[c];
    }
}

// Features of the pair (fiber i, neighbour m), one thread per pair: nine
// floats per neighbour in fiber i's frame.  Slot 0 is neighbour m: its
// relative centre, its orientation u with the canonical sign (u_z > 0, ties
// broken by u_y then u_x; the sign goes to sign[]) and u squared; slots
// 1..15 are the other neighbours, nearest first: relative centre and the six
// products u_a u_b (the sign of their orientation does not change block m).
__global__ void pair_features_kernel(int M, int kp, const double *__restrict__ pos, const double *__restrict__ ori,
                                     const int *__restrict__ knn, float *__restrict__ feat,
                                     float *__restrict__ sign, float *__restrict__ rot) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)M * kp) return;
    const int i = (int)(t / kp), m = (int)(t - (int64_t)i * kp);
    const int *nb = knn + (int64_t)i * kK;
    double E[3][3];
    fiber_frame(pos, ori, i, nb[0], E);
    if (m == 0)
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c) rot[(int64_t)i * 9 + r * 3 + c] = (float)E[r][c];
    const double *xi = pos + 3 * i;
    float *f = feat + t * kIn;
    auto local = [&](int j, double dl[3], double ul[3]) {
        const double d[3] = {pos[3 * j] - xi[0], pos[3 * j + 1] - xi[1], pos[3 * j + 2] - xi[2]};
        const double *tj = ori + 3 * j;
        for (int r = 0; r < 3; ++r) {
            dl[r] = E[r][0] * d[0] + E[r][1] * d[1] + E[r][2] * d[2];
            ul[r] = E[r][0] * tj[0] + E[r][1] * tj[1] + E[r][2] * tj[2];
        }
    };
    double dl[3], ul[3];
    local(nb[m], dl, ul);
    const bool pos_sign = ul[2] > 0.0 || (ul[2] == 0.0 && (ul[1] > 0.0 || (ul[1] == 0.0 && ul[0] >= 0.0)));
    const double s = pos_sign ? 1.0 : -1.0;
    sign[t] = (float)s;
    for (int r = 0; r < 3; ++r) {
        f[r] = (float)dl[r];
        f[3 + r] = (float)(s * ul[r]);
        f[6 + r] = (float)(ul[r] * ul[r]);
    }
    int slot = 1;
    for (int n = 0; n < kK; ++n) {
        if (n == m) continue;
        local(nb[n], dl, ul);
        float *g = f + slot * 9;
        g[0] = (float)dl[0];
        g[1] = (float)dl[1];
        g[2] = (float)dl[2];
        g[3] = (float)(ul[0] * ul[0]);
        g[4] = (float)(ul[1] * ul[1]);
        g[5] = (float)(ul[2] * ul[2]);
        g[6] = (float)(ul[0] * ul[1]);
        g[7] = (float)(ul[0] * ul[2]);
        g[8] = (float)(ul[1] * ul[2]);
        ++slot;
    }
}

// local <-> global pair blocks: B = (R_blk^T O R_blk) D (to_global) or
// O = (R_blk B R_blk^T) D (to_local), R_blk = I_5 (x) R of fiber i, D = the
// pair's sign on the columns of odd Legendre order k (lb = k - 1 even).  One
// thread per pair block; the output of pairs m >= kp is zero.
__global__ void pair_frame_kernel(int M, int kp, const float *__restrict__ rot, const float *__restrict__ sign,
                                  const float *__restrict__ in, int64_t in_stride, float *__restrict__ out,
                                  int64_t out_stride, int to_global) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)M * kPair) return;
    const int i = (int)(t / kPair), m = (int)(t - (int64_t)i * kPair);
    const int64_t q = (int64_t)i * kp + m;  // row of the per-pair arrays (features, MLP output)
    float *Y = out + (to_global ? t : q) * out_stride;
    if (m >= kp) {
        if (to_global)
            for (int e = 0; e < kOut; ++e) Y[e] = 0.f;
        return;
    }
    float R[9];
    for (int e = 0; e < 9; ++e) R[e] = rot[(int64_t)i * 9 + e];
    const float s = sign[q];
    const float *X = in + (to_global ? q : t) * in_stride;
    for (int kb = 0; kb < 5; ++kb)
        for (int lb = 0; lb < 5; ++lb) {
            float O[3][3], T[3][3];
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) O[a][b] = X[(kb * 3 + a) * kNb + lb * 3 + b];
            // to_global: Z = R^T O R ; to_local: Z = R O R^T
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    float acc = 0.f;
                    for (int c = 0; c < 3; ++c) acc += O[a][c] * (to_global ? R[c * 3 + b] : R[b * 3 + c]);
                    T[a][b] = acc;
                }
            const float d = (lb % 2 == 0) ? s : 1.f;
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) {
                    float acc = 0.f;
                    for (int c = 0; c < 3; ++c) acc += (to_global ? R[c * 3 + a] : R[a * 3 + c]) * T[c][b];
                    Y[(kb * 3 + a) * kNb + lb * 3 + b] = d * acc;
                }
        }
}

}  // namespace

// ------------------------------------------------------------------ handle side
namespace {
// neighbours found by knn_kernel (stride kK per fiber) and blocks kept per fiber
int knn_count(const rf_handle *h) { return std::min(kK, h->M - 1); }

rf_status ensure_pair_buffers(rf_handle *h) {
    const int M = h->M, nb = 3 * h->N;
    auto ck = [&](cudaError_t e, const char *what) -> rf_status {
        return e == cudaSuccess ? RF_OK : cuda_fail(h, e, what);
    };
    rf_status s;
    if (!h->Pblocks &&
        (s = ck(cudaMalloc(&h->Pblocks, sizeof(float) * (size_t)M * kPair * nb * nb), "alloc blocks")) != RF_OK)
        return s;
    if (!h->knn && (s = ck(cudaMalloc(&h->knn, sizeof(int) * (size_t)M * kK), "alloc knn")) != RF_OK) return s;
    return RF_OK;
}

rf_status ensure_mlp_buffers(rf_handle *h) {
    const size_t rows = (size_t)h->M * kPair;
    auto ck = [&](cudaError_t e, const char *what) -> rf_status {
        return e == cudaSuccess ? RF_OK : cuda_fail(h, e, what);
    };
    rf_status s;
    if (h->feat) return RF_OK;
    // features, then the frames (9 per fiber) and the pair signs (1 per pair)
    if ((s = ck(cudaMalloc(&h->feat, sizeof(float) * (rows * kIn + (size_t)h->M * 9 + rows)), "alloc")) != RF_OK)
        return s;
    if ((s = ck(cudaMalloc(&h->mlp_h1, sizeof(float) * rows * kHid), "alloc")) != RF_OK) return s;
    if ((s = ck(cudaMalloc(&h->mlp_h2, sizeof(float) * rows * kHid), "alloc")) != RF_OK) return s;
    if ((s = ck(cudaMalloc(&h->mlp_out, sizeof(float) * rows * kOut), "alloc")) != RF_OK) return s;
    return RF_OK;
}

float *feat_rot(rf_handle *h) { return h->feat + (size_t)h->M * kPair * kIn; }
float *feat_sign(rf_handle *h) { return feat_rot(h) + (size_t)h->M * 9; }

cudaError_t launch_knn(rf_handle *h) {
    knn_kernel<<<(h->M + kKnnWarps - 1) / kKnnWarps, kKnnWarps * 32, 0, h->stream>>>(h->M, h->X[h->cur], kK, h->knn);
    h->launches++;
    return cudaGetLastError();
}

// pair features (M x kPair rows), the frames and the signs of the current state
cudaError_t launch_pair_features(rf_handle *h) {
    const int64_t rows = (int64_t)h->M * kPair;
    pair_features_kernel<<<(unsigned)((rows + 127) / 128), 128, 0, h->stream>>>(
        h->M, kPair, h->X[h->cur], h->T[h->cur], h->knn, h->feat, feat_sign(h), feat_rot(h));
    h->launches++;
    return cudaGetLastError();
}
}  // namespace

rf_status build_preconditioner(rf_handle *h) {
    const int M = h->M, nb = 3 * h->N;
    cudaStream_t st = h->stream;
    auto ck = [&](cudaError_t e, const char *what) -> rf_status {
        return e == cudaSuccess ? RF_OK : cuda_fail(h, e, what);
    };
    rf_status s;
    if ((s = ensure_pair_buffers(h)) != RF_OK) return s;
    const int K = knn_count(h);
    if ((s = ck(launch_knn(h), "knn")) != RF_OK) return s;
    h->pc_pairs = 0;
    if (h->p.preconditioner == RF_PC_CLUSTER) {
        const int kc = std::max(1, std::min(h->p.cluster_size, K));
        const int kp = std::min(kPair, kc);
        const int sdim = (kc + 1) * nb;
        const size_t smem = sizeof(float) * (size_t)sdim * (sdim + nb + 1);
        if (smem > 227 * 1024)
            return fail(h, RF_ERR_INVALID_ARG, "cluster_size too large for the shared-memory factorisation");
        int *sing = nullptr;
        if ((s = ck(cudaMalloc(&sing, sizeof(int)), "alloc")) != RF_OK) return s;
        cudaMemsetAsync(sing, 0, sizeof(int), st);
        cudaError_t e;
        if (h->A64) {
            e = cudaFuncSetAttribute(cluster_rows_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem);
            if (e == cudaSuccess)
                cluster_rows_kernel<double><<<M, 256, smem, st>>>(M, nb, h->A64, h->lda, 0, h->knn, kK, kc, kp,
                                                                  h->Pblocks, sing);
        } else if (h->A16lo) {
            e = cudaFuncSetAttribute(cluster_rows_kernel<SplitF32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem);
            if (e == cudaSuccess)
                cluster_rows_kernel<SplitF32><<<M, 256, smem, st>>>(
                    M, nb, reinterpret_cast<const SplitF32 *>(h->A16), h->lda, h->a_plane, h->knn, kK, kc, kp,
                    h->Pblocks, sing);
        } else {
            e = cudaFuncSetAttribute(cluster_rows_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem);
            if (e == cudaSuccess)
                cluster_rows_kernel<float><<<M, 256, smem, st>>>(M, nb, h->A32, h->lda, 0, h->knn, kK, kc, kp,
                                                                 h->Pblocks, sing);
        }
        h->launches++;
        if (e == cudaSuccess) e = cudaGetLastError();
        cudaFree(sing);
        if ((s = ck(e, "cluster inverse")) != RF_OK) return s;
        h->pc_pairs = kp;
        h->pc_ready = true;
        return RF_OK;
    }
    // learned
    if (!h->mlp_loaded || nb != kNb || K < kK) {
        h->pc_ready = false;  // fallback: no preconditioning (block-Jacobi with identity blocks)
        return RF_OK;
    }
    return apply_mlp(h);
}

rf_status apply_mlp(rf_handle *h) {
    const int M = h->M;
    cudaStream_t st = h->stream;
    auto ck = [&](cudaError_t e, const char *what) -> rf_status {
        return e == cudaSuccess ? RF_OK : cuda_fail(h, e, what);
    };
    rf_status s;
    if ((s = ensure_mlp_buffers(h)) != RF_OK) return s;
    if ((s = ck(launch_pair_features(h), "features")) != RF_OK) return s;
    const int rows = M * kPair;
    // inference on the tensor cores (BF16 operands, FP32 accumulation); the
    // FP32 CUDA-core GEMMs remain for training
    const MlpLayout Lw;
    const int P = mlp_tc_padded_rows();
    __nv_bfloat16 *w1 = h->mlp_wtc, *w2 = w1 + (size_t)P * kIn, *w3 = w2 + (size_t)P * kHid;
    if ((s = ck(mlp_tc_forward(w1, h->mlp_w + Lw.b1, w2, h->mlp_w + Lw.b2, w3, h->mlp_w + Lw.b3, rows, kIn, kHid, kOut,
                               h->feat, reinterpret_cast<__nv_bfloat16 *>(h->mlp_h1),
                               reinterpret_cast<__nv_bfloat16 *>(h->mlp_h2), h->mlp_out, h->mlp_err, st),
                "mlp")) != RF_OK)
        return s;
    pair_frame_kernel<<<(unsigned)((rows + 127) / 128), 128, 0, st>>>(M, kPair, feat_rot(h), feat_sign(h), h->mlp_out,
                                                                       kOut, h->Pblocks, kOut, 1);
    h->launches += 4;
    if ((s = ck(cudaGetLastError(), "block frame")) != RF_OK) return s;
    h->pc_pairs = kPair;
    h->pc_ready = true;
    return RF_OK;
}

}  // namespace rf

// ------------------------------------------------------------------ C ABI
using namespace rf;

struct rf_trainer {
    int device = 0;
    cudaStream_t stream = nullptr;
    float *W = nullptr, *G = nullptr, *Mom = nullptr, *Var = nullptr;
    float *X = nullptr, *Y = nullptr;      // dataset
    int64_t count = 0, cap = 0;
    float *bx = nullptr, *by = nullptr;    // a batch
    rf::MlpBatch b{};                      // and its intermediate results
    int bcap = 0;
    int *perm = nullptr;                   // an epoch's order of the samples
    int64_t perm_cap = 0;
    double *sse = nullptr;                 // summed squared error
    int64_t t = 0;
    std::mt19937_64 rng;
};

extern "C" {

int64_t rf_mlp_num_params(void) { return MlpLayout().total; }

rf_status rf_set_mlp_weights(rf_handle *h, const float *weights, int64_t count) {
    if (!h || !weights || count != MlpLayout().total) return fail(h, RF_ERR_INVALID_ARG, "weights: wrong size");
    if (cudaSetDevice(h->device) != cudaSuccess) return fail(h, RF_ERR_CUDA, "cudaSetDevice");
    if (!h->mlp_w && cudaMalloc(&h->mlp_w, sizeof(float) * count) != cudaSuccess)
        return fail(h, RF_ERR_OOM, "alloc weights");
    if (cudaMemcpy(h->mlp_w, weights, sizeof(float) * count, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(h, RF_ERR_CUDA, "upload weights");
    // BF16 copies of W1, W2, W3 with their rows padded to the tensor-core tile
    const MlpLayout Lw;
    const int P = mlp_tc_padded_rows();
    if (!h->mlp_wtc && (cudaMalloc(&h->mlp_wtc, sizeof(__nv_bfloat16) * (size_t)P * (kIn + 2 * kHid)) != cudaSuccess ||
                        cudaMalloc(&h->mlp_err, sizeof(int)) != cudaSuccess))
        return fail(h, RF_ERR_OOM, "alloc weights");
    __nv_bfloat16 *w1 = h->mlp_wtc, *w2 = w1 + (size_t)P * kIn, *w3 = w2 + (size_t)P * kHid;
    if (mlp_tc_pad_weights(h->mlp_w + Lw.w1, kHid, kIn, w1, h->stream) != cudaSuccess ||
        mlp_tc_pad_weights(h->mlp_w + Lw.w2, kHid, kHid, w2, h->stream) != cudaSuccess ||
        mlp_tc_pad_weights(h->mlp_w + Lw.w3, kOut, kHid, w3, h->stream) != cudaSuccess ||
        cudaMemsetAsync(h->mlp_err, 0, sizeof(int), h->stream) != cudaSuccess ||
        cudaStreamSynchronize(h->stream) != cudaSuccess)
        return fail(h, RF_ERR_CUDA, "convert weights");
    h->mlp_loaded = true;
    h->pc_ready = false;
    return RF_OK;
}

rf_status rf_compute_features(rf_handle *h, float *features) {
    if (!h || !features) return fail(h, RF_ERR_INVALID_ARG, "null argument");
    if (h->M <= kK) return fail(h, RF_ERR_INVALID_ARG, "features need more than 16 fibers");
    if (cudaSetDevice(h->device) != cudaSuccess) return fail(h, RF_ERR_CUDA, "cudaSetDevice");
    rf_status s;
    if ((s = ensure_pair_buffers(h)) != RF_OK || (s = ensure_mlp_buffers(h)) != RF_OK) return s;
    cudaError_t e = launch_knn(h);
    if (e == cudaSuccess) e = launch_pair_features(h);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(features, h->feat, sizeof(float) * (size_t)h->M * kPair * kIn, cudaMemcpyDeviceToHost,
                            h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return cuda_fail(h, e, "features");
    return RF_OK;
}

rf_status rf_compute_cluster_targets(rf_handle *h, float *targets) {
    if (!h || !targets) return fail(h, RF_ERR_INVALID_ARG, "null argument");
    if (!h->assembled) return fail(h, RF_ERR_INVALID_ARG, "cluster targets need an assembled system");
    if (3 * h->N != kNb) return fail(h, RF_ERR_INVALID_ARG, "the learned blocks are built for N = 5");
    if (h->M <= kK) return fail(h, RF_ERR_INVALID_ARG, "targets need more than 16 fibers");
    if (h->p.cluster_size < kPair) return fail(h, RF_ERR_INVALID_ARG, "targets need cluster_size >= 8");
    if (cudaSetDevice(h->device) != cudaSuccess) return fail(h, RF_ERR_CUDA, "cudaSetDevice");
    const int saved = h->p.preconditioner;
    h->p.preconditioner = RF_PC_CLUSTER;
    rf_status s = build_preconditioner(h);   // exact coupling blocks into Pblocks
    h->p.preconditioner = saved;
    if (s != RF_OK) return s;
    // the frames and signs of the same state, then the blocks in that frame
    if ((s = ensure_mlp_buffers(h)) != RF_OK) return s;
    const int64_t rows = (int64_t)h->M * kPair;
    cudaError_t e = launch_pair_features(h);
    if (e == cudaSuccess) {
        pair_frame_kernel<<<(unsigned)((rows + 127) / 128), 128, 0, h->stream>>>(
            h->M, kPair, feat_rot(h), feat_sign(h), h->Pblocks, kOut, h->mlp_out, kOut, 0);
        h->launches++;
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(targets, h->mlp_out, sizeof(float) * rows * kOut, cudaMemcpyDeviceToHost, h->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
    if (e != cudaSuccess) return cuda_fail(h, e, "targets");
    if (saved != RF_PC_CLUSTER) h->pc_ready = false;
    return RF_OK;
}

rf_status rf_mlp_predict(int32_t device, const float *weights, const float *features, int64_t count, float *out) {
    if (!weights || !features || !out || count < 1 || count > (1 << 22))
        return fail(nullptr, RF_ERR_INVALID_ARG, "rf_mlp_predict: bad arguments");
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return fail(nullptr, RF_ERR_NO_DEVICE, "no CUDA device");
    }
    const MlpLayout Lw;
    const int P = mlp_tc_padded_rows();
    float *w = nullptr, *x = nullptr, *o = nullptr;
    __nv_bfloat16 *wt = nullptr, *h1 = nullptr, *h2 = nullptr;
    int *err = nullptr;
    cudaStream_t st = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaMalloc(&w, sizeof(float) * Lw.total);
    if (e == cudaSuccess) e = cudaMalloc(&x, sizeof(float) * count * kIn);
    if (e == cudaSuccess) e = cudaMalloc(&o, sizeof(float) * count * kOut);
    if (e == cudaSuccess) e = cudaMalloc(&wt, sizeof(__nv_bfloat16) * (size_t)P * (kIn + 2 * kHid));
    if (e == cudaSuccess) e = cudaMalloc(&h1, sizeof(__nv_bfloat16) * count * kHid);
    if (e == cudaSuccess) e = cudaMalloc(&h2, sizeof(__nv_bfloat16) * count * kHid);
    if (e == cudaSuccess) e = cudaMalloc(&err, sizeof(int));
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(w, weights, sizeof(float) * Lw.total, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(x, features, sizeof(float) * count * kIn, cudaMemcpyHostToDevice, st);
    __nv_bfloat16 *w1 = wt, *w2 = w1 + (size_t)P * kIn, *w3 = w2 + (size_t)P * kHid;
    if (e == cudaSuccess) e = mlp_tc_pad_weights(w + Lw.w1, kHid, kIn, w1, st);
    if (e == cudaSuccess) e = mlp_tc_pad_weights(w + Lw.w2, kHid, kHid, w2, st);
    if (e == cudaSuccess) e = mlp_tc_pad_weights(w + Lw.w3, kOut, kHid, w3, st);
    if (e == cudaSuccess)
        e = mlp_tc_forward(w1, w + Lw.b1, w2, w + Lw.b2, w3, w + Lw.b3, (int)count, kIn, kHid, kOut, x, h1, h2, o, err,
                           st);
    int herr = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, o, sizeof(float) * count * kOut, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    void *ptrs[] = {w, x, o, wt, h1, h2, err};
    for (void *p : ptrs) cudaFree(p);
    if (st) cudaStreamDestroy(st);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "rf_mlp_predict");
    if (herr) return fail(nullptr, RF_ERR_DEVICE_TIMEOUT, "rf_mlp_predict: tensor-core wait timed out");
    return RF_OK;
}

rf_status rf_trainer_create(int32_t device, uint64_t seed, rf_trainer **out) {
    if (!out) return fail(nullptr, RF_ERR_INVALID_ARG, "out is null");
    *out = nullptr;
    if (cudaSetDevice(device) != cudaSuccess) {
        cudaGetLastError();
        return fail(nullptr, RF_ERR_NO_DEVICE, "no CUDA device");
    }
    rf_trainer *t = new rf_trainer;
    t->device = device;
    t->rng.seed(seed);
    const int64_t P = MlpLayout().total;
    bool ok = cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&t->W, sizeof(float) * P) == cudaSuccess && cudaMalloc(&t->G, sizeof(float) * P) == cudaSuccess &&
              cudaMalloc(&t->Mom, sizeof(float) * P) == cudaSuccess && cudaMalloc(&t->Var, sizeof(float) * P) == cudaSuccess &&
              cudaMalloc(&t->sse, sizeof(double)) == cudaSuccess;
    if (!ok) {
        rf_trainer_destroy(t);
        return fail(nullptr, RF_ERR_OOM, "trainer allocation");
    }
    // He-uniform initial weights, small output layer, zero biases
    const MlpLayout L;
    std::vector<float> w(P, 0.f);
    auto fill = [&](int64_t off, int fan_out, int fan_in, float gain) {
        std::uniform_real_distribution<float> u(-1.f, 1.f);
        const float a = gain * std::sqrt(6.f / fan_in);
        for (int64_t e = 0; e < (int64_t)fan_out * fan_in; ++e) w[off + e] = a * u(t->rng);
    };
    fill(L.w1, kHid, kIn, 1.f);
    fill(L.w2, kHid, kHid, 1.f);
    fill(L.w3, kOut, kHid, 0.1f);
    cudaMemcpy(t->W, w.data(), sizeof(float) * P, cudaMemcpyHostToDevice);
    cudaMemset(t->Mom, 0, sizeof(float) * P);
    cudaMemset(t->Var, 0, sizeof(float) * P);
    *out = t;
    return RF_OK;
}

rf_status rf_trainer_destroy(rf_trainer *t) {
    if (!t) return RF_ERR_INVALID_ARG;
    cudaSetDevice(t->device);
    void *ptrs[] = {t->W, t->G, t->Mom, t->Var, t->X, t->Y, t->bx, t->perm, t->sse};
    for (void *p : ptrs) cudaFree(p);
    if (t->stream) cudaStreamDestroy(t->stream);
    delete t;
    return RF_OK;
}

rf_status rf_trainer_add_samples(rf_trainer *t, const float *features, const float *targets, int64_t count) {
    if (!t || !features || !targets || count < 1) return fail(nullptr, RF_ERR_INVALID_ARG, "bad samples");
    cudaSetDevice(t->device);
    if (t->count + count > t->cap) {
        int64_t ncap = std::max<int64_t>(t->cap * 2, t->count + count);
        float *nx = nullptr, *ny = nullptr;
        if (cudaMalloc(&nx, sizeof(float) * ncap * kIn) != cudaSuccess ||
            cudaMalloc(&ny, sizeof(float) * ncap * kOut) != cudaSuccess) {
            cudaFree(nx);
            return fail(nullptr, RF_ERR_OOM, "dataset");
        }
        if (t->count) {
            cudaMemcpy(nx, t->X, sizeof(float) * t->count * kIn, cudaMemcpyDeviceToDevice);
            cudaMemcpy(ny, t->Y, sizeof(float) * t->count * kOut, cudaMemcpyDeviceToDevice);
        }
        cudaFree(t->X);
        cudaFree(t->Y);
        t->X = nx;
        t->Y = ny;
        t->cap = ncap;
    }
    if (cudaMemcpy(t->X + t->count * kIn, features, sizeof(float) * count * kIn, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(t->Y + t->count * kOut, targets, sizeof(float) * count * kOut, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(nullptr, RF_ERR_CUDA, "upload samples");
    t->count += count;
    return RF_OK;
}

namespace {
// Buffers of a batch, one allocation (its first float is bx).
bool ensure_batch(rf_trainer *t, int B) {
    if (B <= t->bcap) return true;
    cudaFree(t->bx);
    const int64_t n = B;
    const int64_t sizes[] = {n * kIn, n * kOut, n * kHid, n * kHid, n * kMlpOutLd, n * kHid, n * kHid,
                             mlp_slices(B) * MlpLayout().total, 2 * (int64_t)mlp_loss_parts(B)};
    float *sse = nullptr;
    float **to[] = {&t->bx, &t->by, &t->b.h1, &t->b.h2, &t->b.dO, &t->b.dh2, &t->b.dh1, &t->b.part, &sse};
    int64_t total = 0;
    for (int64_t s : sizes) total += (s + 3) / 4 * 4;  // each on 16 bytes
    float *p = nullptr;
    t->bcap = 0;
    const bool ok = cudaMalloc(&p, sizeof(float) * total) == cudaSuccess;
    if (!ok) cudaGetLastError();
    for (int i = 0; i < 9; ++i) {
        *to[i] = ok ? p : nullptr;
        if (ok) p += (sizes[i] + 3) / 4 * 4;
    }
    t->b.sse = reinterpret_cast<double *>(sse);
    if (ok) t->bcap = B;
    return ok;
}
}  // namespace

rf_status rf_trainer_train(rf_trainer *t, int32_t epochs, int32_t batch, float lr, float *loss) {
    if (!t || epochs < 1 || batch < 1 || t->count < 1) return fail(nullptr, RF_ERR_INVALID_ARG, "bad training call");
    cudaSetDevice(t->device);
    if (!ensure_batch(t, batch)) return fail(nullptr, RF_ERR_OOM, "batch buffers");
    if (t->count > t->perm_cap) {
        cudaFree(t->perm);
        t->perm = nullptr;
        t->perm_cap = 0;
        if (cudaMalloc(&t->perm, sizeof(int) * t->count) != cudaSuccess) {
            cudaGetLastError();
            return fail(nullptr, RF_ERR_OOM, "sample order");
        }
        t->perm_cap = t->count;
    }
    // An epoch is queued without waiting for the device: the order of the
    // samples goes up once, the squared error is summed on the device.
    std::vector<int> perm(t->count);
    double sse = 0.0;
    for (int ep = 0; ep < epochs; ++ep) {
        for (int64_t i = 0; i < t->count; ++i) perm[i] = (int)i;
        std::shuffle(perm.begin(), perm.end(), t->rng);
        cudaError_t e = cudaMemcpyAsync(t->perm, perm.data(), sizeof(int) * t->count, cudaMemcpyHostToDevice, t->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(t->sse, 0, sizeof(double), t->stream);
        for (int64_t b0 = 0; b0 < t->count && e == cudaSuccess; b0 += batch) {
            const int B = (int)std::min<int64_t>(batch, t->count - b0);
            e = mlp_gather(B, t->perm + b0, t->X, t->Y, t->bx, t->by, t->stream);
            if (e == cudaSuccess) e = mlp_gradient(t->b, t->W, B, t->bx, t->by, t->G, t->sse, t->stream);
            t->t += 1;
            const float b1 = 0.9f, b2 = 0.999f;
            const float c1 = 1.f - std::pow(b1, (float)t->t), c2 = 1.f - std::pow(b2, (float)t->t);
            if (e == cudaSuccess) e = mlp_adam(t->W, t->G, t->Mom, t->Var, lr, b1, b2, c1, c2, 1e-8f, t->stream);
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&sse, t->sse, sizeof(double), cudaMemcpyDeviceToHost, t->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
        if (e != cudaSuccess) return cuda_fail(nullptr, e, "training step");
    }
    if (loss) *loss = (float)(sse / ((double)t->count * kOut));
    return RF_OK;
}

rf_status rf_trainer_get_weights(rf_trainer *t, float *weights) {
    if (!t || !weights) return fail(nullptr, RF_ERR_INVALID_ARG, "null argument");
    cudaSetDevice(t->device);
    if (cudaMemcpy(weights, t->W, sizeof(float) * MlpLayout().total, cudaMemcpyDeviceToHost) != cudaSuccess)
        return fail(nullptr, RF_ERR_CUDA, "download weights");
    return RF_OK;
}

rf_status rf_trainer_set_weights(rf_trainer *t, const float *weights) {
    if (!t || !weights) return fail(nullptr, RF_ERR_INVALID_ARG, "null argument");
    cudaSetDevice(t->device);
    if (cudaMemcpy(t->W, weights, sizeof(float) * MlpLayout().total, cudaMemcpyHostToDevice) != cudaSuccess)
        return fail(nullptr, RF_ERR_CUDA, "upload weights");
    return RF_OK;
}

rf_status rf_trainer_loss_grad(rf_trainer *t, const float *features, const float *targets, int64_t count, float *loss,
                               float *grad) {
    if (!t || !features || !targets || count < 1 || count > (1 << 20))
        return fail(nullptr, RF_ERR_INVALID_ARG, "bad arguments");
    cudaSetDevice(t->device);
    if (!ensure_batch(t, (int)count)) return fail(nullptr, RF_ERR_OOM, "batch buffers");
    double sse = 0.0;
    cudaError_t e = cudaMemcpyAsync(t->bx, features, sizeof(float) * count * kIn, cudaMemcpyHostToDevice, t->stream);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(t->by, targets, sizeof(float) * count * kOut, cudaMemcpyHostToDevice, t->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(t->sse, 0, sizeof(double), t->stream);
    if (e == cudaSuccess) e = mlp_gradient(t->b, t->W, (int)count, t->bx, t->by, t->G, t->sse, t->stream);
    if (e == cudaSuccess && grad)
        e = cudaMemcpyAsync(grad, t->G, sizeof(float) * MlpLayout().total, cudaMemcpyDeviceToHost, t->stream);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&sse, t->sse, sizeof(double), cudaMemcpyDeviceToHost, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "loss/grad");
    if (loss) *loss = (float)(sse / ((double)count * kOut));
    return RF_OK;
}

}  // extern "C"
