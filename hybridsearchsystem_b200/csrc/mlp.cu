// mlp.cu -- the learned threshold predictor: a small MLP (features -> 2 hidden layers with GELU ->
// one output, the predicted K-th filtered score), trained and run by these kernels.
//
//   forward   Z1 = X W1 + b1, A1 = gelu(Z1), Z2 = A1 W2 + b2, A2 = gelu(Z2), y = A2 w3 + b3
//   backward  from dL/dy: the gradients of every parameter (GEMMs with transposed operands, GELU'
//             from the stored pre-activations, bias gradients as column sums)
//   adam      one Adam step over the flat parameter vector
// FP32 throughout. The products of a training step are small (512 x 397 x 256 at most at its usual batch,
// 0.4 GFLOP in all, 6 us at the FP32 rate), so the step is bound by latency: few CTAs, dependent launches
// and the load latency of each k step. Hence five launches instead of fourteen (each pass's elementwise
// work in its epilogue, independent products side by side in one grid, bias gradients from the tiles that
// a product already stages), 32 x 32 output tiles (at least 100 CTAs) and operands copied by cp.async
// two or three k steps ahead; the gradients' products, whose sums may take any order, split k four ways inside a
// CTA. The forward pass keeps one sum per output over k ascending. At a batch of 512, 397 features and
// 256 hidden units the kernels took 432 us (64 x 64 tiles on 4 to 32 CTAs) and take 61 us from the first's
// start to the last's end.
#include <algorithm>

#include "hss_device.cuh"
#include "hss_kernels.h"

namespace hss {
namespace {

__device__ inline float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ inline float gelu_grad(float z) {
    // d/dz [z Phi(z)] = Phi(z) + z phi(z)
    const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return cdf + z * pdf;
}

constexpr int kTile = 32;          // output tile: 32 x 32, 2 x 4 outputs per thread of a group
constexpr int kTileK = 32;         // k per stage
constexpr int kGroup = 128;        // threads that share one k range
constexpr int kPitch = kTile + 4;  // staged rows of 36 floats: 16-byte reads
constexpr int kStageFloats = 2 * kTile * kPitch;
constexpr int kGradSplit = 4;      // k split of the gradients' products
constexpr int kGradThreads = kGroup * kGradSplit;
constexpr int kFwdStages = 4, kGradStages = 3;
constexpr size_t kFwdSmem = static_cast<size_t>(kFwdStages) * kStageFloats * sizeof(float);
constexpr size_t kGradSmem = static_cast<size_t>(kGradSplit) * kGradStages * kStageFloats * sizeof(float);

// One product's operands: C[M][N] = op(A) op(B) over K.
struct Product {
    const float *A, *B;
    int M, N, K, lda, ldb;
};

// min(words, `width`) floats (width 4: 16-byte aligned addresses; 1: any), zeros in the rest of width.
template <int width>
__device__ __forceinline__ void copy_async(float* smem, const float* gmem, int words) {
    const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const int bytes = 4 * max(0, min(words, width));
    if (width == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(gmem), "r"(bytes) : "memory");
}

// A 32 x 32 block of a row-major matrix [rows][cols] (pitch ld) from (r0, c0), to smem rows of kPitch;
// zeros outside the matrix. 16-byte copies where the matrix allows them.
__device__ __forceinline__ void copy_block(float* smem, const float* M, int rows, int cols, int ld, int r0, int c0,
                                           int t, bool vec) {
    if (vec) {
#pragma unroll
        for (int i = 0; i < kTile * kTileK / 4 / kGroup; ++i) {
            const int f = t + kGroup * i, r = f / 8, c = f % 8 * 4;
            const bool in = r0 + r < rows && c0 + c < cols;
            copy_async<4>(smem + r * kPitch + c, in ? M + static_cast<int64_t>(r0 + r) * ld + c0 + c : M,
                          in ? cols - c0 - c : 0);
        }
    } else {
#pragma unroll
        for (int i = 0; i < kTile * kTileK / kGroup; ++i) {
            const int f = t + kGroup * i, r = f / 32, c = f % 32;
            const bool in = r0 + r < rows && c0 + c < cols;
            copy_async<1>(smem + r * kPitch + c, in ? M + static_cast<int64_t>(r0 + r) * ld + c0 + c : M, in ? 1 : 0);
        }
    }
}

__device__ __forceinline__ bool rows_of_16_bytes(const float* M, int ld) {
    return (reinterpret_cast<uintptr_t>(M) & 15u) == 0 && (ld & 3) == 0;
}

// The tile at (m0, n0) of one product, into acc of group 0's threads: thread t has rows
// 2 (t / 8) + {0, 1} and columns tile_col(t % 8, {0..3}). KS groups of 128 threads take every KS-th stage
// of k and are summed in group order. op(A)(m, k) = TA ? A[k * lda + m] : A[m * lda + k], likewise
// op(B)(k, n) = TB ? B[n * ldb + k] : B[k * ldb + n]; both are staged as they lie, and four k at a time
// are read from an operand whose rows run along k. With colsum (TB false), thread t < 32 of group 0 also
// gets the sum over k of op(B)'s column n0 + t in *colsum.
template <bool TB>
__device__ __forceinline__ int tile_col(int tx, int j) {
    return TB ? tx + 8 * j : 4 * tx + j;  // TB: the 8 rows a read takes are neighbours (distinct banks)
}

template <bool TA, bool TB, int KS, int ST>
__device__ __forceinline__ void product_tile(const Product& P, int m0, int n0, float* smem, float (&acc)[2][4],
                                             float* colsum) {
    const int g = threadIdx.x / kGroup, t = threadIdx.x % kGroup;
    const int tx = t % 8, ty = t / 8;
    float* ring = smem + g * ST * kStageFloats;
    const int chunks = (P.K + kTileK - 1) / kTileK;
    const int steps = (chunks + KS - 1) / KS;
    const bool vecA = rows_of_16_bytes(P.A, P.lda), vecB = rows_of_16_bytes(P.B, P.ldb);
    auto load = [&](int step) {
        float* sA = ring + (step % ST) * kStageFloats;
        float* sB = sA + kTile * kPitch;
        const int k0 = (step * KS + g) * kTileK;
        copy_block(sA, P.A, TA ? P.K : P.M, TA ? P.M : P.K, P.lda, TA ? k0 : m0, TA ? m0 : k0, t, vecA);
        copy_block(sB, P.B, TB ? P.N : P.K, TB ? P.K : P.N, P.ldb, TB ? n0 : k0, TB ? k0 : n0, t, vecB);
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    float cs = 0.0f;
    for (int s = 0; s < ST - 1; ++s) {
        if (s < steps) load(s);
        commit();
    }
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();  // the stage has landed, and the one loaded next has been read by every thread
        if (step + ST - 1 < steps) load(step + ST - 1);
        commit();
        const float* sA = ring + (step % ST) * kStageFloats;
        const float* sB = sA + kTile * kPitch;
#pragma unroll 4
        for (int k = 0; k < kTileK; k += 4) {
            float a[2][4], b[4][4];  // [row][k], [k][column]
            if (TA) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const float2 x = *reinterpret_cast<const float2*>(sA + (k + u) * kPitch + 2 * ty);
                    a[0][u] = x.x;
                    a[1][u] = x.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float4 x = *reinterpret_cast<const float4*>(sA + (2 * ty + i) * kPitch + k);
                    a[i][0] = x.x;
                    a[i][1] = x.y;
                    a[i][2] = x.z;
                    a[i][3] = x.w;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float4 x = *reinterpret_cast<const float4*>(TB ? sB + tile_col<TB>(tx, u) * kPitch + k
                                                                     : sB + (k + u) * kPitch + 4 * tx);
                if (TB) {
                    b[0][u] = x.x;
                    b[1][u] = x.y;
                    b[2][u] = x.z;
                    b[3][u] = x.w;
                } else {
                    b[u][0] = x.x;
                    b[u][1] = x.y;
                    b[u][2] = x.z;
                    b[u][3] = x.w;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i][u], b[u][j], acc[i][j]);
        }
        if (colsum && t < kTile) {
#pragma unroll 8
            for (int kk = 0; kk < kTileK; ++kk) cs += sB[kk * kPitch + t];
        }
    }
    if (KS > 1) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        float* part = smem;  // [KS - 1][9][kGroup]
        if (g > 0) {
#pragma unroll
            for (int j = 0; j < 8; ++j) part[((g - 1) * 9 + j) * kGroup + t] = acc[j / 4][j % 4];
            part[((g - 1) * 9 + 8) * kGroup + t] = cs;
        }
        __syncthreads();
        if (g == 0) {
#pragma unroll
            for (int s = 0; s < KS - 1; ++s) {
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j / 4][j % 4] += part[(s * 9 + j) * kGroup + t];
                cs += part[(s * 9 + 8) * kGroup + t];
            }
        }
    }
    if (colsum) *colsum = cs;
}

// fn(index into C, row, column, value) for the outputs of a tile that lie inside [M][N] (group 0 only).
template <bool TB, class Fn>
__device__ __forceinline__ void store_tile(const Product& P, int m0, int n0, const float (&acc)[2][4], Fn fn) {
    if (threadIdx.x >= kGroup) return;
    const int tx = threadIdx.x % 8, ty = threadIdx.x / 8;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int m = m0 + 2 * ty + i;
        if (m >= P.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tile_col<TB>(tx, j);
            if (n < P.N) fn(static_cast<int64_t>(m) * P.N + n, n, acc[i][j]);
        }
    }
}

__device__ __forceinline__ void tile_of(int64_t tile, int N, int* m0, int* n0) {
    const int across = (N + kTile - 1) / kTile;
    *m0 = static_cast<int>(tile / across) * kTile;
    *n0 = static_cast<int>(tile % across) * kTile;
}

// A hidden layer of the training pass: Z = A W + b, act = gelu(Z).
__global__ void __launch_bounds__(kGroup) layer_forward_kernel(Product P, const float* bias,
                                                               float* Z, float* act) {
    extern __shared__ __align__(16) float gsm[];
    launch_dependents();
    wait_for_previous();
    int m0, n0;
    tile_of(blockIdx.x, P.N, &m0, &n0);
    float acc[2][4];
    product_tile<false, false, 1, kFwdStages>(P, m0, n0, gsm, acc, nullptr);
    store_tile<false>(P, m0, n0, acc, [&](int64_t at, int n, float v) {
        const float z = v + bias[n];
        Z[at] = z;
        act[at] = gelu(z);
    });
}

// The output layer, the loss and the way back to the second hidden layer, for kHeadRows rows:
// y = A2 w3 + b3 (each row's sum over k ascending), the loss's gradient dy and term, and
// dZ2 = (dy w3^T) * gelu'(Z2). tau = 0: mean squared error, dy = 2 (y - t) / B, term (y - t)^2. tau in
// (0, 1): the pinball loss of the tau-quantile, term tau (t - y) when t >= y and (1 - tau) (y - t)
// otherwise, dy = (y > t ? 1 - tau : -tau) / B (the network then predicts a conditional tau-quantile of
// the target).
constexpr int kHeadRows = 8;
constexpr int kHeadT = 256;
constexpr int kHeadK = 256;

__global__ void __launch_bounds__(kHeadT) head_kernel(const float* A2, const float* Z2,
                                                      const float* w3, const float* b3,
                                                      const float* target, int B, int H, float tau,
                                                      float* dy, float* term,
                                                      float* dZ2) {
    __shared__ float sa[kHeadRows][kHeadK + 1];
    __shared__ float sw[kHeadK];
    __shared__ float sdy[kHeadRows];
    launch_dependents();
    wait_for_previous();
    const int r0 = blockIdx.x * kHeadRows, t = threadIdx.x;
    const int rows = min(kHeadRows, B - r0);
    float acc = 0.0f;
    for (int k0 = 0; k0 < H; k0 += kHeadK) {
        const int kc = min(kHeadK, H - k0);
        if (t < kc) sw[t] = w3[k0 + t];
#pragma unroll
        for (int r = 0; r < kHeadRows; ++r)
            if (t < kc && r < rows) sa[r][t] = A2[static_cast<int64_t>(r0 + r) * H + k0 + t];
        __syncthreads();
        if (t < rows) {
#pragma unroll 16
            for (int k = 0; k < kc; ++k) acc = fmaf(sa[t][k], sw[k], acc);
        }
        __syncthreads();
    }
    if (t < rows) {
        const float d = acc + b3[0] - target[r0 + t];
        float g, l;
        if (tau <= 0.0f) {
            g = 2.0f * d / static_cast<float>(B);
            l = d * d;
        } else {
            g = (d > 0.0f ? 1.0f - tau : -tau) / static_cast<float>(B);
            l = d > 0.0f ? (1.0f - tau) * d : -tau * d;
        }
        sdy[t] = g;
        dy[r0 + t] = g;
        term[r0 + t] = l;
    }
    __syncthreads();
    for (int j = t; j < H; j += kHeadT) {
        const float w = w3[j];
#pragma unroll
        for (int r = 0; r < kHeadRows; ++r)
            if (r < rows) {
                const int64_t at = static_cast<int64_t>(r0 + r) * H + j;
                dZ2[at] = sdy[r] * w * gelu_grad(Z2[at]);
            }
    }
}

// Gradients of the output and second hidden layer, one grid: tiles [0, tilesA) dZ1 = (dZ2 W2^T) *
// gelu'(Z1), then tilesW of dW2 = A1^T dZ2 (those of the first 32 rows also db2, the columns' sums of
// dZ2), then blocks of 32 outputs of dw3 = A2^T dy (the first also db3 = sum dy).
__global__ void __launch_bounds__(kGradThreads) grad_hidden_kernel(Product dA, const float* Z1,
                                                                   float* dZ1, int64_t tilesA, Product dW,
                                                                   float* gW2, float* gb2,
                                                                   int64_t tilesW, const float* A2,
                                                                   const float* dy, int B, int H,
                                                                   float* gw3, float* gb3) {
    extern __shared__ __align__(16) float gsm[];
    launch_dependents();
    wait_for_previous();
    int64_t tile = blockIdx.x;
    int m0, n0;
    float acc[2][4];
    if (tile < tilesA) {
        tile_of(tile, dA.N, &m0, &n0);
        product_tile<false, true, kGradSplit, kGradStages>(dA, m0, n0, gsm, acc, nullptr);
        store_tile<true>(dA, m0, n0, acc, [&](int64_t at, int, float v) { dZ1[at] = v * gelu_grad(Z1[at]); });
        return;
    }
    tile -= tilesA;
    if (tile < tilesW) {
        tile_of(tile, dW.N, &m0, &n0);
        float cs = 0.0f;
        product_tile<true, false, kGradSplit, kGradStages>(dW, m0, n0, gsm, acc, m0 == 0 ? &cs : nullptr);
        store_tile<false>(dW, m0, n0, acc, [&](int64_t at, int, float v) { gW2[at] = v; });
        if (m0 == 0 && threadIdx.x < kTile && n0 + static_cast<int>(threadIdx.x) < dW.N) gb2[n0 + threadIdx.x] = cs;
        return;
    }
    tile -= tilesW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = static_cast<int>(tile) * 32 + lane;
    constexpr int kWarps = kGradThreads / 32;
    float s = 0.0f, sd = 0.0f;
#pragma unroll 4
    for (int m = warp; m < B; m += kWarps) {
        const float g = dy[m];
        if (j < H) s = fmaf(A2[static_cast<int64_t>(m) * H + j], g, s);
        sd += g;
    }
    gsm[warp * 32 + lane] = s;
    if (lane == 0) gsm[kWarps * 32 + warp] = sd;
    __syncthreads();
    if (warp == 0) {
        float v = 0.0f, d = 0.0f;
        for (int w = 0; w < kWarps; ++w) {
            v += gsm[w * 32 + lane];
            d += gsm[kWarps * 32 + w];
        }
        if (j < H) gw3[j] = v;
        if (tile == 0 && lane == 0) gb3[0] = d;
    }
}

// dW1 = X^T dZ1, db1 = the columns' sums of dZ1.
__global__ void __launch_bounds__(kGradThreads) grad_input_kernel(Product dW, float* gW1,
                                                                  float* gb1) {
    extern __shared__ __align__(16) float gsm[];
    launch_dependents();
    wait_for_previous();
    int m0, n0;
    tile_of(blockIdx.x, dW.N, &m0, &n0);
    float acc[2][4];
    float cs = 0.0f;
    product_tile<true, false, kGradSplit, kGradStages>(dW, m0, n0, gsm, acc, m0 == 0 ? &cs : nullptr);
    store_tile<false>(dW, m0, n0, acc, [&](int64_t at, int, float v) { gW1[at] = v; });
    if (m0 == 0 && threadIdx.x < kTile && n0 + static_cast<int>(threadIdx.x) < dW.N) gb1[n0 + threadIdx.x] = cs;
}

// Inference forward pass fused into one launch: a CTA takes kFwdRows feature rows, thread j computes
// hidden unit j of both layers for all of them, and thread r < kFwdRows the output of row r. Every sum
// runs over k in ascending order with fmaf, the bias added after, as layer_forward_kernel and head_kernel
// do: the outputs equal the training pass's (launch_train_gradients) bit for bit.
constexpr int kFwdRows = 4;
constexpr int kFwdUnroll = 64;  // weight loads in flight per thread

__global__ void mlp_forward_kernel(const float* __restrict__ X, int B, int D, int H, const float* __restrict__ P,
                                   float* __restrict__ y) {
    extern __shared__ float fsm[];
    float* xs = fsm;                  // [kFwdRows][D]
    float* a1 = xs + kFwdRows * D;    // [kFwdRows][H]
    float* a2 = a1 + kFwdRows * H;    // [kFwdRows][H]
    const int r0 = blockIdx.x * kFwdRows;
    const int rows = min(kFwdRows, B - r0);
    for (int i = threadIdx.x; i < kFwdRows * D; i += blockDim.x) {
        const int r = i / D;
        xs[i] = r < rows ? X[static_cast<int64_t>(r0 + r) * D + i % D] : 0.0f;
    }
    __syncthreads();
    const float* W1 = P;
    const float* b1 = W1 + static_cast<int64_t>(D) * H;
    const float* W2 = b1 + H;
    const float* b2 = W2 + static_cast<int64_t>(H) * H;
    const float* w3 = b2 + H;
    const float* b3 = w3 + H;
    const int j = threadIdx.x;
    // acc[r] += in[r][k] * W[k][j] for k ascending; the weights of kFwdUnroll k's are loaded before
    // they are used, so that many loads are in flight (the loop is otherwise bound by load latency)
    // (the last block is partial: its loads and sums stop at K, a uniform condition)
    auto layer = [&](const float* __restrict__ W, const float* in, int K, float (&acc)[kFwdRows]) {
        for (int k = 0; k < K; k += kFwdUnroll) {
            float w[kFwdUnroll];
#pragma unroll
            for (int u = 0; u < kFwdUnroll; ++u) w[u] = k + u < K ? __ldg(W + static_cast<int64_t>(k + u) * H + j) : 0.0f;
#pragma unroll
            for (int u = 0; u < kFwdUnroll; ++u) {
                if (k + u < K) {
#pragma unroll
                    for (int r = 0; r < kFwdRows; ++r) acc[r] = fmaf(in[r * K + k + u], w[u], acc[r]);
                }
            }
        }
    };
    if (j < H) {
        float acc[kFwdRows] = {};
        layer(W1, xs, D, acc);
#pragma unroll
        for (int r = 0; r < kFwdRows; ++r) a1[r * H + j] = gelu(acc[r] + b1[j]);
    }
    __syncthreads();
    if (j < H) {
        float acc[kFwdRows] = {};
        layer(W2, a1, H, acc);
#pragma unroll
        for (int r = 0; r < kFwdRows; ++r) a2[r * H + j] = gelu(acc[r] + b2[j]);
    }
    __syncthreads();
    if (j < rows) {
        float acc = 0.0f;
        for (int k = 0; k < H; ++k) acc = fmaf(a2[j * H + k], w3[k], acc);
        y[r0 + j] = acc + b3[0];
    }
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, int64_t n, float lr, float b1, float b2, float eps, float c1,
                            float c2) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// Features of one query (row q of X, din columns): [ q * sqrt(dim) | per posting row: 1 + log10
// density / 4 for the rows of the query's filter, 0 elsewhere | log10 selectivity / 4 | log10 K / 3 |
// 1 | the doc sample's best score | its K-th best score (-2 when absent) | log10(filtered sample
// docs + 1) / 5 ].
__global__ void features_kernel(FeatureLaunch L) {
    const uint32_t q = blockIdx.x;
    float* x = L.x + static_cast<uint64_t>(q) * L.din;
    const float s = sqrtf(static_cast<float>(L.dim));
    for (uint32_t i = threadIdx.x; i < L.din; i += blockDim.x) {
        float v = 0.0f;
        if (i < L.dim) v = L.qry[static_cast<uint64_t>(q) * L.dim + i] * s;
        x[i] = v;
    }
    __syncthreads();
    const uint32_t o0 = L.opnd_off[q], o1 = L.opnd_off[q + 1];
    for (uint32_t j = o0 + threadIdx.x; j < o1; j += blockDim.x) {
        const uint32_t r = L.opnd_row[j];
        if (r < L.rows) x[L.dim + r] = 1.0f + log10f(fmaxf(L.row_density[r], 1e-9f)) * 0.25f;
    }
    if (threadIdx.x == 0) {
        const float sel = fmaxf(static_cast<float>(L.pass_count[q]), 1.0f) / static_cast<float>(L.doc_num);
        const float* st = L.stats + static_cast<uint64_t>(q) * kSampleStats;
        float* t = x + L.dim + L.rows;
        t[0] = log10f(sel) * 0.25f;
        t[1] = log10f(fmaxf(static_cast<float>(L.topk[q]), 1.0f)) / 3.0f;
        t[2] = 1.0f;
        for (uint32_t j = 0; j < kSampleRanks; ++j) t[3 + j] = st[j];
        t[3 + kSampleRanks] = st[kSampleRanks];
        t[4 + kSampleRanks] = log10f(st[kSampleRanks + 1] + 1.0f) * 0.2f;
    }
}

// theta[q] = max(proven threshold, predicted K-th score (y * scale + shift) minus the margin and the
// query's error bound), the proven one kept in theta_proven. A doc of the true top K then clears
// theta whenever the prediction minus the margin is at most the true K-th score. A query whose filter
// passes at most kLearnedMinPass * K docs keeps its proven threshold: its candidates are few whatever
// the threshold, and its K-th score is the hardest to predict. So does a query whose doc sample held
// fewer than kLearnedMinSample filtered docs (its sample rank features are missing). fmaxf drops a
// NaN prediction.
// theta_model may alias y (each thread reads, then writes, its own element).
__global__ void predict_theta_kernel(const float* y, const float* __restrict__ eps,
                                     const uint32_t* __restrict__ pass_count, const uint32_t* __restrict__ topk,
                                     const float* __restrict__ stats, uint32_t nq, float scale, float shift,
                                     float margin, float* theta, float* theta_proven, float* theta_model) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nq) return;
    const float t1 = theta[q];
    const bool use = static_cast<uint64_t>(pass_count[q]) > static_cast<uint64_t>(kLearnedMinPass) * topk[q] &&
                     stats[static_cast<uint64_t>(q) * kSampleStats + kSampleRanks + 1] >= kLearnedMinSample;
    const float t = use ? fmaxf(t1, __fsub_rd(__fsub_rd(fmaf(y[q], scale, shift), margin), eps[q])) : t1;
    theta_proven[q] = t1;
    theta[q] = t;
    theta_model[q] = t;
}

}  // namespace

cudaError_t launch_train_gradients(const TrainLaunch& L, cudaStream_t stream) {
    if (L.B <= 0) return cudaSuccess;
    if (!(L.tau >= 0.0f && L.tau < 1.0f)) return cudaErrorInvalidValue;
    const int B = L.B, D = L.D, H = L.H;
    auto tiles = [](int m, int n) {
        return static_cast<int64_t>((m + kTile - 1) / kTile) * ((n + kTile - 1) / kTile);
    };
    const float* W1 = L.P;
    const float* b1 = W1 + static_cast<int64_t>(D) * H;
    const float* W2 = b1 + H;
    const float* b2 = W2 + static_cast<int64_t>(H) * H;
    const float* w3 = b2 + H;
    const float* b3 = w3 + H;
    float* gW1 = L.G;
    float* gb1 = gW1 + static_cast<int64_t>(D) * H;
    float* gW2 = gb1 + H;
    float* gb2 = gW2 + static_cast<int64_t>(H) * H;
    float* gw3 = gb2 + H;
    float* gb3 = gw3 + H;
    const int64_t tF = tiles(B, H), tW2 = tiles(H, H), tW1 = tiles(D, H), tw3 = (H + 31) / 32;
    if (tF + tW2 + tw3 > 0x7fffffff || tW1 > 0x7fffffff) return cudaErrorInvalidValue;
    for (const void* k : {reinterpret_cast<const void*>(grad_hidden_kernel),
                          reinterpret_cast<const void*>(grad_input_kernel)}) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(kGradSmem));
        if (e != cudaSuccess) return e;
    }
    const dim3 gF(static_cast<unsigned>(tF));
    cudaError_t e = launch_dependent(layer_forward_kernel, gF, kGroup, kFwdSmem, stream, 1,
                                     Product{L.X, W1, B, H, D, D, H}, b1, L.Z1, L.A1);
    if (e == cudaSuccess)
        e = launch_dependent(layer_forward_kernel, gF, kGroup, kFwdSmem, stream, 1, Product{L.A1, W2, B, H, H, H, H},
                             b2, L.Z2, L.A2);
    if (e == cudaSuccess)
        e = launch_dependent(head_kernel, dim3((B + kHeadRows - 1) / kHeadRows), kHeadT, 0, stream, 1, L.A2, L.Z2, w3,
                             b3, L.T, B, H, L.tau, L.dy, L.term, L.dZ2);
    if (e == cudaSuccess)
        e = launch_dependent(grad_hidden_kernel, dim3(static_cast<unsigned>(tF + tW2 + tw3)), kGradThreads, kGradSmem,
                             stream, 1, Product{L.dZ2, W2, B, H, H, H, H}, L.Z1, L.dZ1, tF,
                             Product{L.A1, L.dZ2, H, H, B, H, H}, gW2, gb2, tW2, L.A2, L.dy, B, H, gw3, gb3);
    if (e == cudaSuccess)
        e = launch_dependent(grad_input_kernel, dim3(static_cast<unsigned>(tW1)), kGradThreads, kGradSmem, stream, 1,
                             Product{L.X, L.dZ1, D, H, B, D, H}, gW1, gb1);
    return e;
}

cudaError_t launch_mlp_forward(const float* X, int B, int D, int H, const float* P, float* y, cudaStream_t stream) {
    if (B <= 0) return cudaSuccess;
    const int threads = ((std::max(H, kFwdRows) + 31) / 32) * 32;
    const size_t smem = static_cast<size_t>(kFwdRows) * (D + 2 * H) * sizeof(float);
    if (threads > 1024 || smem > 48 * 1024) return cudaErrorInvalidValue;
    mlp_forward_kernel<<<(B + kFwdRows - 1) / kFwdRows, threads, smem, stream>>>(X, B, D, H, P, y);
    return cudaGetLastError();
}

cudaError_t launch_adam(float* p, const float* g, float* m, float* v, int64_t n, float lr, float b1, float b2,
                        float eps, int step, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    const float c1 = 1.0f - powf(b1, static_cast<float>(step));
    const float c2 = 1.0f - powf(b2, static_cast<float>(step));
    adam_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(p, g, m, v, n, lr, b1, b2, eps, c1, c2);
    return cudaGetLastError();
}

cudaError_t launch_features(const FeatureLaunch& L, cudaStream_t stream) {
    if (L.nq == 0) return cudaSuccess;
    if (L.din < L.dim + L.rows + kFeatureTail || !L.stats) return cudaErrorInvalidValue;
    features_kernel<<<L.nq, 128, 0, stream>>>(L);
    return cudaGetLastError();
}

cudaError_t launch_predict_theta(const float* y, const float* eps, const uint32_t* pass_count, const uint32_t* topk,
                                 const float* stats, uint32_t nq, float scale, float shift, float margin,
                                 float* theta, float* theta_proven, float* theta_model, cudaStream_t stream) {
    if (nq == 0) return cudaSuccess;
    predict_theta_kernel<<<(nq + 127) / 128, 128, 0, stream>>>(y, eps, pass_count, topk, stats, nq, scale, shift,
                                                               margin, theta, theta_proven, theta_model);
    return cudaGetLastError();
}

}  // namespace hss
