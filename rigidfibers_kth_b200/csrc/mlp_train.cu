// mlp_train.cu - one training step's kernels of the preconditioner MLP (FP32):
// forward, squared-error loss, backward and Adam on a batch.
//
// The layers (144 -> 256 -> 256 -> 225, ReLU) at the usual batch of 512 rows
// are small: 0.45 GFLOP in all.  What bounds a step is parallelism and the
// number of dependent launches, so
//   * the forward and data-gradient products run in 32 x 32 tiles while 64 x 64
//     ones would leave SMs idle, four by four outputs per thread, the k range
//     split over four groups of a CTA's threads (one group: 15 us a layer);
//   * bias, ReLU, the loss with its gradient (the last layer's output is never
//     stored) and the ReLU masks of the backward pass are epilogues;
//   * the three weight gradients and the bias sums are one launch over (tile,
//     slice of the batch), the slices' partial sums added in order by a second.
// Seven launches per gradient.  Before: thirteen, with weight-gradient grids of
// 16 CTAs over the whole batch (85 us each) and one CTA per bias sum (32 us).
// Gradient at 512 rows, kernels cold: 540 -> 69 us, the call with its pageable
// copies of 1.4 MB 625 -> 290 us; 8192 rows 4650 -> 1140 us; a training epoch of
// 98 such batches (order uploaded once, loss summed on the device, no wait per
// batch) 40 -> 7.3 ms.
// All sums in FP32 (the loss in FP64) in an order that depends on the batch
// size alone.
#include <algorithm>

#include "mlp_train.h"

namespace rf {
namespace {

constexpr int kBK = 16;

enum Epilogue { kBiasRelu, kLoss, kMask };

struct LayerArgs {
    int m, n, k;             // C m x n = A (m x k, rows of lda) op(B)
    const float *A;
    int lda;
    const float *B;          // BT: B(k, j) = B[j ldb + k], else B[k ldb + j]
    int ldb;
    float *C;
    int ldc;
    const float *bias;       // kBiasRelu, kLoss
    const float *mask;       // kMask: C = 0 where mask (ld ldc) <= 0
    const float *target;     // kLoss (m x n): C = 2 (o - target) / (m n), sse[CTA] = sum (o - target)^2
    double *sse;
};

// a kBK x T tile of an operand into shared memory, [k][row]: K contiguous in
// memory (transposed on the way) or rows contiguous; zero outside
template <int T, int THREADS, bool KCONT>
struct TileLoad {
    static constexpr int kPer = T * kBK / 4 / THREADS;
    float4 r[kPer];
    __device__ __forceinline__ void load(const float *p, int ld, int row0, int rows, int k0, int k1) {
        const int tid = threadIdx.x % THREADS;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int e = tid + u * THREADS;
            r[u] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (KCONT) {
                const int i = row0 + e / (kBK / 4), k = k0 + 4 * (e % (kBK / 4));
                if (i < rows && k < k1) r[u] = *reinterpret_cast<const float4 *>(p + (int64_t)i * ld + k);
                if (k + 1 >= k1) r[u].y = 0.f;
                if (k + 2 >= k1) r[u].z = 0.f;
                if (k + 3 >= k1) r[u].w = 0.f;
            } else {
                const int i = row0 + 4 * (e % (T / 4)), k = k0 + e / (T / 4);
                if (i < rows && k < k1) r[u] = *reinterpret_cast<const float4 *>(p + (int64_t)k * ld + i);
                if (i + 1 >= rows) r[u].y = 0.f;
                if (i + 2 >= rows) r[u].z = 0.f;
                if (i + 3 >= rows) r[u].w = 0.f;
            }
        }
    }
    __device__ __forceinline__ void store(float (*s)[T + 4]) const {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int e = threadIdx.x % THREADS + u * THREADS;
            if (KCONT) {
                const int i = e / (kBK / 4), k = 4 * (e % (kBK / 4));
                s[k][i] = r[u].x;
                s[k + 1][i] = r[u].y;
                s[k + 2][i] = r[u].z;
                s[k + 3][i] = r[u].w;
            } else {
                *reinterpret_cast<float4 *>(&s[e / (T / 4)][4 * (e % (T / 4))]) = r[u];
            }
        }
    }
};

// acc += the product of the staged tiles: thread (ty, tx) owns rows 4 ty .. and
// columns 4 tx ..
template <int T>
__device__ __forceinline__ void tile_product(const float (*sa)[T + 4], const float (*sb)[T + 4], int ty, int tx,
                                             float (&acc)[4][4], float *asum) {
#pragma unroll
    for (int k = 0; k < kBK; ++k) {
        const float4 a4 = *reinterpret_cast<const float4 *>(&sa[k][4 * ty]);
        const float4 b4 = *reinterpret_cast<const float4 *>(&sb[k][4 * tx]);
        const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (asum) asum[u] += a[u];
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(a[u], b[v], acc[u][v]);
        }
    }
}

// T x T tiles by G groups of T^2 / 16 threads, group q taking every G-th block
// of k and the groups' sums added in order; the next tiles travel while these
// are used
template <int T, int G, bool BT, int EPI>
__global__ void __launch_bounds__(G * T * T / 16) layer_kernel(LayerArgs g) {
    constexpr int THREADS = T * T / 16;
    struct Stage {
        float a[2][kBK][T + 4], b[2][kBK][T + 4];
    };
    __shared__ __align__(16) Stage s_st[G];
    __shared__ double s_red[THREADS / 32];
    static_assert(sizeof(Stage) >= sizeof(float) * T * T, "a group's sums fit its tiles");
    const int grp = G > 1 ? threadIdx.x / THREADS : 0;
    const int tid = threadIdx.x % THREADS, tx = tid % (T / 4), ty = tid / (T / 4);
    const int i0 = blockIdx.y * T, j0 = blockIdx.x * T;
    Stage &st = s_st[grp];
    TileLoad<T, THREADS, true> la;
    TileLoad<T, THREADS, BT> lb;
    float acc[4][4] = {};
    la.load(g.A, g.lda, i0, g.m, grp * kBK, g.k);
    lb.load(g.B, g.ldb, j0, g.n, grp * kBK, g.k);
    la.store(st.a[0]);
    lb.store(st.b[0]);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < g.k; k0 += G * kBK) {  // the same number of steps for every group
        const bool more = k0 + G * kBK < g.k;
        if (more) {
            la.load(g.A, g.lda, i0, g.m, k0 + (G + grp) * kBK, g.k);
            lb.load(g.B, g.ldb, j0, g.n, k0 + (G + grp) * kBK, g.k);
        }
        tile_product<T>(st.a[buf], st.b[buf], ty, tx, acc, nullptr);
        if (more) {
            buf ^= 1;
            la.store(st.a[buf]);
            lb.store(st.b[buf]);
        }
        __syncthreads();
    }
    if (G > 1) {
        float *own = reinterpret_cast<float *>(&st) + 16 * tid;
        if (grp > 0) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                *reinterpret_cast<float4 *>(own + 4 * u) = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
        }
        __syncthreads();
        if (grp > 0) return;
        for (int q = 1; q < G; ++q) {
            const float *p = reinterpret_cast<const float *>(&s_st[q]) + 16 * tid;
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] += p[4 * u + v];
        }
    }
    double sse = 0.0;
    const float scale = EPI == kLoss ? (float)((int64_t)g.m * g.n) : 1.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = i0 + 4 * ty + u;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int j = j0 + 4 * tx + v;
            if (i >= g.m || j >= g.n) continue;
            float *c = g.C + (int64_t)i * g.ldc + j;
            if (EPI == kBiasRelu) *c = fmaxf(acc[u][v] + g.bias[j], 0.f);
            if (EPI == kMask) *c = g.mask[(int64_t)i * g.ldc + j] <= 0.f ? 0.f : acc[u][v];
            if (EPI == kLoss) {
                const float d = (acc[u][v] + g.bias[j]) - g.target[(int64_t)i * g.n + j];
                *c = 2.f * d / scale;
                sse += (double)d * d;
            }
        }
    }
    if (EPI == kLoss) {
#pragma unroll
        for (int o = 16; o; o >>= 1) sse += __shfl_xor_sync(0xffffffffu, sse, o);
        if (tid % 32 == 0) s_red[tid / 32] = sse;
        asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");  // the first group alone is left
        if (tid == 0) {
            double s = 0.0;
            for (int q = 0; q < THREADS / 32; ++q) s += s_red[q];
            g.sse[blockIdx.y * gridDim.x + blockIdx.x] = s;
        }
    }
}

// Weight gradients dW = dY^T H (rows of the batch summed) and bias gradients
// (column sums of dY) of the three layers: blockIdx.x a 64 x 64 tile of one of
// them, blockIdx.y a slice of the batch.
struct GradArgs {
    int rows, per;           // batch rows; rows per slice
    struct {
        const float *dY, *H; // rows x m (ld ldy), rows x n (ld ldh)
        int m, n, ldy, ldh, tile0, tx;   // first tile of the layer, tiles across
        int64_t w, b;        // offsets of the layer's weights and biases
    } l[3];
    float *part;             // [slices][params]
    int64_t params;
};
__global__ void __launch_bounds__(256) weight_grad_kernel(GradArgs g) {
    constexpr int T = 64;
    __shared__ __align__(16) float sa[2][kBK][T + 4], sb[2][kBK][T + 4];
    const int tid = threadIdx.x, tx = tid % (T / 4), ty = tid / (T / 4);
    const int which = (int)blockIdx.x >= g.l[2].tile0 ? 2 : (int)blockIdx.x >= g.l[1].tile0 ? 1 : 0;
    const auto l = which == 2 ? g.l[2] : which == 1 ? g.l[1] : g.l[0];
    const int t = blockIdx.x - l.tile0, i0 = t / l.tx * T, j0 = t % l.tx * T;
    const int k0 = blockIdx.y * g.per, k1 = min(g.rows, k0 + g.per);
    TileLoad<T, 256, false> la, lb;
    float acc[4][4] = {}, asum[4] = {};
    la.load(l.dY, l.ldy, i0, l.m, k0, k1);
    lb.load(l.H, l.ldh, j0, l.n, k0, k1);
    la.store(sa[0]);
    lb.store(sb[0]);
    __syncthreads();
    int buf = 0;
    for (int k = k0; k < k1; k += kBK) {
        const bool more = k + kBK < k1;
        if (more) {
            la.load(l.dY, l.ldy, i0, l.m, k + kBK, k1);
            lb.load(l.H, l.ldh, j0, l.n, k + kBK, k1);
        }
        tile_product<T>(sa[buf], sb[buf], ty, tx, acc, asum);
        if (more) {
            buf ^= 1;
            la.store(sa[buf]);
            lb.store(sb[buf]);
        }
        __syncthreads();
    }
    float *out = g.part + (int64_t)blockIdx.y * g.params;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int i = i0 + 4 * ty + u;
        if (i >= l.m) continue;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int j = j0 + 4 * tx + v;
            if (j < l.n) out[l.w + (int64_t)i * l.n + j] = acc[u][v];
        }
        if (j0 == 0 && tx == 0) out[l.b + i] = asum[u];
    }
}

// gradient = the slices' partial sums in order; the first CTA also adds the
// loss partials to *sse
__global__ void __launch_bounds__(256) grad_reduce_kernel(const float *part, int slices, int64_t params, float *G,
                                                          const double *sse_part, int nsse, double *sse) {
    const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (e < params) {
        float s = 0.f;
        for (int q = 0; q < slices; ++q) s += part[(int64_t)q * params + e];
        G[e] = s;
    }
    if (blockIdx.x == 0) {
        __shared__ double sh[256];
        double s = 0.0;
        for (int q = threadIdx.x; q < nsse; q += 256) s += sse_part[q];
        sh[threadIdx.x] = s;
        __syncthreads();
        for (int o = 128; o > 0; o >>= 1) {
            if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) *sse += sh[0];
    }
}

__global__ void adam_kernel(int64_t cnt, float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                            float *__restrict__ v, float lr, float b1, float b2, float c1, float c2, float eps) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x) {
        const float gi = g[e];
        const float mi = b1 * m[e] + (1.f - b1) * gi;
        const float vi = b2 * v[e] + (1.f - b2) * gi * gi;
        m[e] = mi;
        v[e] = vi;
        w[e] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

// rows idx[0..rows) of the dataset into the batch
__global__ void gather_kernel(int rows, const int *__restrict__ idx, const float *__restrict__ X,
                              const float *__restrict__ Y, float *__restrict__ bx, float *__restrict__ by) {
    const int r = blockIdx.x;
    const int64_t s = idx[r];
    for (int c = threadIdx.x; c < kMlpIn / 4; c += blockDim.x)
        reinterpret_cast<float4 *>(bx + (int64_t)r * kMlpIn)[c] = reinterpret_cast<const float4 *>(X + s * kMlpIn)[c];
    for (int c = threadIdx.x; c < kMlpOut; c += blockDim.x) by[(int64_t)r * kMlpOut + c] = Y[s * kMlpOut + c];
}

// 64 x 64 tiles once they fill the GPU, 32 x 32 before (at 512 rows 64 x 64 tiles
// are 32 CTAs: 36 us for the second layer in the ncu launch list, 32 x 32 8.7 us)
constexpr int kFullGpu = 148;
template <bool BT, int EPI>
cudaError_t layer(const LayerArgs &g, int *ctas, cudaStream_t st) {
    auto grid = [&](int T) { return dim3((unsigned)((g.n + T - 1) / T), (unsigned)((g.m + T - 1) / T)); };
    const dim3 g64 = grid(64), g32 = grid(32);
    if ((int64_t)g64.x * g64.y >= kFullGpu) {
        layer_kernel<64, 1, BT, EPI><<<g64, 256, 0, st>>>(g);
        *ctas = g64.x * g64.y;
    } else {
        layer_kernel<32, 4, BT, EPI><<<g32, 256, 0, st>>>(g);
        *ctas = g32.x * g32.y;
    }
    return cudaGetLastError();
}

}  // namespace

int mlp_slices(int rows) { return std::max(1, std::min(8, rows / 128)); }

int mlp_loss_parts(int rows) { return ((rows + 31) / 32) * ((kMlpOut + 31) / 32); }

cudaError_t mlp_gradient(const MlpBatch &b, const float *W, int rows, const float *X, const float *Y, float *G,
                         double *sse, cudaStream_t st) {
    const MlpLayout L;
    int ctas = 0, nsse = 0;
    LayerArgs g{};
    g.m = rows;
    g.n = kMlpHid; g.k = kMlpIn; g.A = X; g.lda = kMlpIn; g.B = W + L.w1; g.ldb = kMlpIn;
    g.C = b.h1; g.ldc = kMlpHid; g.bias = W + L.b1;
    cudaError_t e = layer<true, kBiasRelu>(g, &ctas, st);
    if (e != cudaSuccess) return e;
    g.k = kMlpHid; g.A = b.h1; g.lda = kMlpHid; g.B = W + L.w2; g.ldb = kMlpHid; g.C = b.h2; g.bias = W + L.b2;
    if ((e = layer<true, kBiasRelu>(g, &ctas, st)) != cudaSuccess) return e;
    g.n = kMlpOut; g.A = b.h2; g.B = W + L.w3; g.C = b.dO; g.ldc = kMlpOutLd; g.bias = W + L.b3; g.target = Y;
    g.sse = b.sse;
    if ((e = layer<true, kLoss>(g, &nsse, st)) != cudaSuccess) return e;
    // dH2 = dO W3 and dH1 = dH2 W2 behind the ReLU
    g = LayerArgs{};
    g.m = rows;
    g.n = kMlpHid; g.k = kMlpOut; g.A = b.dO; g.lda = kMlpOutLd; g.B = W + L.w3; g.ldb = kMlpHid;
    g.C = b.dh2; g.ldc = kMlpHid; g.mask = b.h2;
    if ((e = layer<false, kMask>(g, &ctas, st)) != cudaSuccess) return e;
    g.k = kMlpHid; g.A = b.dh2; g.lda = kMlpHid; g.B = W + L.w2; g.C = b.dh1; g.mask = b.h1;
    if ((e = layer<false, kMask>(g, &ctas, st)) != cudaSuccess) return e;
    GradArgs w{};
    w.rows = rows;
    const int slices = mlp_slices(rows);
    w.per = ((rows + slices - 1) / slices + kBK - 1) / kBK * kBK;
    w.part = b.part;
    w.params = L.total;
    int tiles = 0;
    auto add = [&](int i, const float *dY, int ldy, int m, const float *H, int ldh, int n, int64_t wo, int64_t bo) {
        w.l[i] = {dY, H, m, n, ldy, ldh, tiles, (n + 63) / 64, wo, bo};
        tiles += (m + 63) / 64 * ((n + 63) / 64);
    };
    add(0, b.dO, kMlpOutLd, kMlpOut, b.h2, kMlpHid, kMlpHid, L.w3, L.b3);
    add(1, b.dh2, kMlpHid, kMlpHid, b.h1, kMlpHid, kMlpHid, L.w2, L.b2);
    add(2, b.dh1, kMlpHid, kMlpHid, X, kMlpIn, kMlpIn, L.w1, L.b1);
    const int used = (rows + w.per - 1) / w.per;
    weight_grad_kernel<<<dim3(tiles, used), 256, 0, st>>>(w);
    grad_reduce_kernel<<<(unsigned)((L.total + 255) / 256), 256, 0, st>>>(b.part, used, L.total, G, b.sse, nsse, sse);
    return cudaGetLastError();
}

cudaError_t mlp_gather(int rows, const int *idx, const float *X, const float *Y, float *bx, float *by,
                       cudaStream_t st) {
    gather_kernel<<<rows, 128, 0, st>>>(rows, idx, X, Y, bx, by);
    return cudaGetLastError();
}

cudaError_t mlp_adam(float *W, const float *G, float *m, float *v, float lr, float b1, float b2, float c1, float c2,
                     float eps, cudaStream_t st) {
    adam_kernel<<<256, 256, 0, st>>>(MlpLayout().total, W, G, m, v, lr, b1, b2, c1, c2, eps);
    return cudaGetLastError();
}

}  // namespace rf
