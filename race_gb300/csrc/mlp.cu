// Multilayer perceptron of the parameter tuner: forward pass, mean-squared-
// error gradients and Adam updates as hand-written CUDA kernels (FP32).
//
// Network: in -> hidden (ReLU) -> ... (hiddenLayers times) -> out, every
// layer y = x W^T + b with W stored row-major [outDim][inDim]. Parameters
// are one flat array: for each layer W then b. The tuner's network is small
// (34 inputs, 3 x 128 hidden, 1 output) and its batches are some hundreds to
// thousands of rows: a product is a few million multiply-adds, so launches and
// the latency of each bound the time, not arithmetic. Forward pass and data
// gradients are therefore one kernel that holds the whole network in shared
// memory (kResident), all layers' weight and bias gradients and the loss
// another (kWeightGrad), which writes the caller's copy as well. Loss and
// gradients of 239 rows, on the GPU and per call: one kernel per product (16
// launches) 146 and 222 us; forward and backward kernels that fetch the weights
// tile by tile and 32 x 32 gradient tiles 33 and 77 us; now 18.5 and 44-51 us
// (512 rows 83 -> 54, 4,096: 131 -> 100, 65,536: 1,179 -> 883). Outputs alone,
// 239 rows: 14.4 -> 10.3 us.
// Networks that do not fit in shared memory take the tiles (kForward: a block
// takes a few rows through all layers, weights in tiles fetched one ahead
// across the layer boundaries; kBackward), networks wider than kFusedDim or
// deeper than kFusedLayers, and wide ones with few rows (byProducts), the
// products one by one (kGemm: 32 x 32 output tiles, 16-deep k slices).
// Each output sums its terms in order with fmaf in either form, so results do
// not depend on the grid; above kGradRows rows the weight gradients are summed
// in chunks of rows, added in order (kGradReduce). The loss reduction runs in
// one block in a fixed order (deterministic).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace race {

namespace {

constexpr int kT = 32;   // output tile
constexpr int kK = 16;   // k slice

enum Epilogue { EPI_NONE = 0, EPI_BIAS = 1, EPI_BIAS_RELU = 2, EPI_RELU_MASK = 3 };

// C[M][N] = op(A)[M][K] op(B)[K][N]; op(A)[m][k] = TA ? A[k*lda+m] : A[m*lda+k],
// op(B)[k][n] = TB ? B[n*ldb+k] : B[k*ldb+n]. Epilogues: + bias[n]; + bias
// then ReLU; multiply by (mask[m*ldc+n] > 0) (gradient through a ReLU whose
// output is mask).
template <bool TA, bool TB>
__global__ void __launch_bounds__(256) kGemm(int M, int N, int K, const float *__restrict__ A, int lda,
                                             const float *__restrict__ B, int ldb, float *__restrict__ C, int ldc,
                                             int epi, const float *__restrict__ bias, const float *__restrict__ mask) {
    __shared__ float sA[kK][kT + 1];
    __shared__ float sB[kK][kT + 1];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16 x 16 threads, 2 x 2 outputs each
    const int m0 = blockIdx.y * kT, n0 = blockIdx.x * kT;
    float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    for (int k0 = 0; k0 < K; k0 += kK) {
        for (int i = threadIdx.x; i < kK * kT; i += 256) {
            const int kk = i / kT, mm = i % kT;
            const int m = m0 + mm, k = k0 + kk;
            sA[kk][mm] = (m < M && k < K) ? (TA ? A[(size_t)k * lda + m] : A[(size_t)m * lda + k]) : 0.f;
            const int n = n0 + mm;
            sB[kk][mm] = (n < N && k < K) ? (TB ? B[(size_t)n * ldb + k] : B[(size_t)k * ldb + n]) : 0.f;
        }
        __syncthreads();
        const int kEnd = min(kK, K - k0);
        for (int kk = 0; kk < kEnd; ++kk) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) acc[i][j] = fmaf(sA[kk][ty + 16 * i], sB[kk][tx + 16 * j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int m = m0 + ty + 16 * i, n = n0 + tx + 16 * j;
            if (m >= M || n >= N) continue;
            float v = acc[i][j];
            if (epi == EPI_BIAS || epi == EPI_BIAS_RELU) v += bias[n];
            if (epi == EPI_BIAS_RELU) v = fmaxf(v, 0.f);
            if (epi == EPI_RELU_MASK && !(mask[(size_t)m * ldc + n] > 0.f)) v = 0.f;
            C[(size_t)m * ldc + n] = v;
        }
}

// db[n] = sum_m dY[m][n], in order of m.
__global__ void kColSum(int M, int N, const float *__restrict__ dY, float *__restrict__ db) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    float s = 0.f;
    for (int m = 0; m < M; ++m) s += dY[(size_t)m * N + n];
    db[n] = s;
}

// Mean squared error over B x O outputs: loss = sum (y-t)^2 / (B O);
// dY = 2 (y - t) / (B O). One block, fixed reduction order.
__global__ void __launch_bounds__(256) kMse(int count, const float *__restrict__ y, const float *__restrict__ t,
                                            float *__restrict__ dY, float *__restrict__ loss) {
    __shared__ float part[256];
    float s = 0.f;
    const float scale = 2.f / (float)count;
    for (int i = threadIdx.x; i < count; i += 256) {
        const float d = y[i] - t[i];
        dY[i] = scale * d;
        s = fmaf(d, d, s);
    }
    part[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) part[threadIdx.x] += part[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = part[0] / (float)count;
}

// ---- fused passes
constexpr int kFusedLayers = 16;  // layers (hidden + 1) of the fused kernels' layer table
constexpr int kFusedDim = 1024;   // widest layer: the rows of two layers fit in shared memory
// Weight tile: 128 results x 64 summed terms, 32 values a thread in flight.
// A tile costs about one L2 round trip (the sums take less), so deep tiles
// mean fewer of them.
constexpr int kTileN = 128, kTileK = 64, kTileVals = kTileN * kTileK / 256;
constexpr size_t kTileBytes = 2 * sizeof(float) * kTileK * (kTileN + 1);
constexpr size_t kResidentBytes = 227 * 1024;  // shared memory of one block, all of it
constexpr int kResidentSms = 152;
constexpr int kGradRows = 512;    // rows summed in one chain per weight gradient
constexpr int kGradChunk = 256;   // rows of a chunk beyond that (at most kGradChunks chunks)
constexpr int kGradChunks = 64;

struct NetView {
    int layers;
    int dimIn[kFusedLayers], dimOut[kFusedLayers];
    const float *w[kFusedLayers], *b[kFusedLayers];
    float *act[kFusedLayers];    // outputs of each layer (B x dimOut), null: not kept
    float *delta[kFusedLayers];  // gradients of each layer's outputs before its ReLU
    float *dw[kFusedLayers], *db[kFusedLayers];
};

// The weight tiles of a pass in the order a block needs them: per layer the
// tiles of kTileN results, each over its kTileK-term slices. Forward: results
// are the layer's outputs; backward (layers last..1): its inputs.
struct TileWalk {
    int l, n0, k0;
};
template <bool BACK>
__device__ __forceinline__ int tileN(const NetView &v, int l) { return BACK ? v.dimIn[l] : v.dimOut[l]; }
template <bool BACK>
__device__ __forceinline__ int tileK(const NetView &v, int l) { return BACK ? v.dimOut[l] : v.dimIn[l]; }
template <bool BACK>
__device__ __forceinline__ bool lastLayer(const NetView &v, int l) { return BACK ? l < 1 : l >= v.layers; }
template <bool BACK>
__device__ __forceinline__ void nextTile(const NetView &v, TileWalk &t) {
    t.k0 += kTileK;
    if (t.k0 < tileK<BACK>(v, t.l)) return;
    t.k0 = 0;
    t.n0 += kTileN;
    if (t.n0 < tileN<BACK>(v, t.l)) return;
    t.n0 = 0;
    t.l += BACK ? -1 : 1;
}

// A thread's values of a tile, term by term (forward: W[n][k] along k, so
// that a warp reads consecutive k; backward: W[k][n] along n).
template <bool BACK>
__device__ __forceinline__ void loadTile(const NetView &v, const TileWalk &t, float (&r)[kTileVals]) {
    const int N = tileN<BACK>(v, t.l), K = tileK<BACK>(v, t.l);
    const float *w = v.w[t.l];
#pragma unroll
    for (int i = 0; i < kTileVals; ++i) {
        const int e = i * 256 + threadIdx.x;
        const int n = t.n0 + (BACK ? e % kTileN : e / kTileK), k = t.k0 + (BACK ? e / kTileN : e % kTileK);
        r[i] = n < N && k < K ? w[BACK ? (size_t)k * N + n : (size_t)n * K + k] : 0.f;
    }
}
template <bool BACK>
__device__ __forceinline__ void storeTile(float (*sw)[kTileN + 1], const float (&r)[kTileVals]) {
#pragma unroll
    for (int i = 0; i < kTileVals; ++i) {
        const int e = i * 256 + threadIdx.x;
        sw[BACK ? e / kTileN : e % kTileK][BACK ? e % kTileN : e / kTileK] = r[i];
    }
}

// One pass over the layers for R rows a block: 128 result columns x two halves
// of the rows per tile. `finish(l, n, row, sum)` turns a layer's sum into the
// value the next layer reads. sx holds the current and the next layer's rows
// (stride D, a multiple of 4); cur selects the current one.
template <bool BACK, int R, typename F>
__device__ __forceinline__ void layerPass(const NetView &v, float (*sw)[kTileK][kTileN + 1], float *sx, int D,
                                          F &&finish) {
    constexpr int H = R / 2;
    const int col = threadIdx.x % kTileN, half = threadIdx.x / kTileN;
    int cur = 0, buf = 0;
    TileWalk t{BACK ? v.layers - 1 : 0, 0, 0}, ahead = t;
    float w[kTileVals], acc[H];
    if (!lastLayer<BACK>(v, t.l)) loadTile<BACK>(v, t, w);
    while (!lastLayer<BACK>(v, t.l)) {
        storeTile<BACK>(sw[buf], w);
        __syncthreads();  // the tile, and before a layer's first one its rows
        nextTile<BACK>(v, ahead);
        if (!lastLayer<BACK>(v, ahead.l)) loadTile<BACK>(v, ahead, w);  // in flight during the sums
        if (t.k0 == 0)
#pragma unroll
            for (int i = 0; i < H; ++i) acc[i] = 0.f;
        const float *x = sx + (size_t)cur * R * D + (size_t)half * H * D + t.k0;
        const int kEnd = min(kTileK, tileK<BACK>(v, t.l) - t.k0);
        int k = 0;
#pragma unroll 4
        for (; k + 4 <= kEnd; k += 4) {
            const float w0 = sw[buf][k][col], w1 = sw[buf][k + 1][col], w2 = sw[buf][k + 2][col],
                        w3 = sw[buf][k + 3][col];
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const float4 q = *(const float4 *)(x + i * D + k);
                acc[i] = fmaf(q.w, w3, fmaf(q.z, w2, fmaf(q.y, w1, fmaf(q.x, w0, acc[i]))));
            }
        }
        for (; k < kEnd; ++k)
#pragma unroll
            for (int i = 0; i < H; ++i) acc[i] = fmaf(x[i * D + k], sw[buf][k][col], acc[i]);
        if (t.k0 + kTileK >= tileK<BACK>(v, t.l) && t.n0 + col < tileN<BACK>(v, t.l))
#pragma unroll
            for (int i = 0; i < H; ++i)
                sx[(size_t)(cur ^ 1) * R * D + (size_t)(half * H + i) * D + t.n0 + col] =
                    finish(t.l, t.n0 + col, half * H + i, acc[i]);
        if (ahead.l != t.l) cur ^= 1;
        t = ahead;
        buf ^= 1;
    }
}

// All layers of R rows: activations to v.act (and the outputs to y if given).
template <int R>
__global__ void __launch_bounds__(256) kForward(NetView v, const float *__restrict__ X, int B, int D, float *y) {
    extern __shared__ __align__(16) float smem[];
    auto sw = (float(*)[kTileK][kTileN + 1]) smem;
    float *sx = smem + kTileBytes / sizeof(float);
    const int m0 = blockIdx.x * R, in = v.dimIn[0];
    for (int i = threadIdx.x; i < R * in; i += 256) {
        const int r = i / in, k = i % in;
        sx[(size_t)r * D + k] = m0 + r < B ? X[(size_t)(m0 + r) * in + k] : 0.f;
    }
    layerPass<false, R>(v, sw, sx, D, [&](int l, int n, int r, float s) {
        s += v.b[l][n];
        if (l + 1 < v.layers) s = fmaxf(s, 0.f);
        if (m0 + r < B) {
            const size_t o = (size_t)(m0 + r) * v.dimOut[l] + n;
            if (v.act[l]) v.act[l][o] = s;
            if (y && l + 1 == v.layers) y[o] = s;
        }
        return s;
    });
}

// Output gradients 2 (y - t) / (B O), then the data gradients of all layers
// for R rows.
template <int R>
__global__ void __launch_bounds__(256) kBackward(NetView v, const float *__restrict__ T, int B, int D) {
    extern __shared__ __align__(16) float smem[];
    auto sw = (float(*)[kTileK][kTileN + 1]) smem;
    float *sx = smem + kTileBytes / sizeof(float);
    const int m0 = blockIdx.x * R, last = v.layers - 1, out = v.dimOut[last], count = B * out;
    const float *y = v.act[last];
    const float scale = 2.f / (float)count;
    for (int i = threadIdx.x; i < R * out; i += 256) {
        const int r = i / out, n = i % out;
        const size_t o = (size_t)(m0 + r) * out + n;
        float d = 0.f;
        if (m0 + r < B) v.delta[last][o] = d = scale * (y[o] - T[o]);
        sx[(size_t)r * D + n] = d;
    }
    layerPass<true, R>(v, sw, sx, D, [&](int l, int n, int r, float s) {
        if (m0 + r < B) {
            const size_t o = (size_t)(m0 + r) * v.dimIn[l] + n;
            if (!(v.act[l - 1][o] > 0.f)) s = 0.f;
            v.delta[l - 1][o] = s;
        }
        return s;
    });
}

// 4- and 16-byte asynchronous copies to shared memory; !on writes zeros.
__device__ __forceinline__ void copy4(float *dst, const float *src, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(on ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy16(float *dst, const float *src, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(on ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copyCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// At most `left` of the latest groups may still be on their way (3 and more count as 3).
__device__ __forceinline__ void copyWait(int left) {
    if (left >= 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
    else if (left == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (left == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Floats between two rows of a layer's weights in shared memory: whole
// float4s, an odd number of them, so that neither a warp reading one float4
// of 32 rows (forward) nor 32 values of one row (backward) meets a bank twice
// in a quarter.
__host__ __device__ inline int weightStride(int K) { return 4 * (((K + 3) / 4) | 1); }
__host__ __device__ inline int layerFloats(int K, int N) { return N * weightStride(K) + ((N + 3) & ~3); }

// acc[i] += sum of x[i][k] w(k..k+3) over whole groups of four terms, in
// order; returns the number of terms. Sixteen terms' operands are read before
// the first multiply-add (8 and 4 where a thread has more rows, which hide the
// reads): 128 terms of one result took 2,450 cycles four at a time, 800 so.
// A float4 that the whole warp reads costs shared memory as much as 32
// different ones, so fewer rows a block are faster while they fit on the GPU.
template <int H, typename W>
__device__ __forceinline__ int termSums(float (&acc)[H], const float *x, int D, int K, W &&weight) {
    constexpr int S = H <= 2 ? 4 : H <= 4 ? 2 : 1;
    int k = 0;
    auto some = [&](auto groups) {
        constexpr int G = decltype(groups)::value;
        float4 w[G], q[G][H];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            w[g] = weight(k + 4 * g);
#pragma unroll
            for (int i = 0; i < H; ++i) q[g][i] = *(const float4 *)(x + i * D + k + 4 * g);
        }
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int i = 0; i < H; ++i)
                acc[i] = fmaf(q[g][i].w, w[g].w,
                              fmaf(q[g][i].z, w[g].z, fmaf(q[g][i].y, w[g].y, fmaf(q[g][i].x, w[g].x, acc[i]))));
        k += 4 * G;
    };
    while (k + 4 * S <= K) some(std::integral_constant<int, S>{});
    while (k + 4 <= K) some(std::integral_constant<int, 1>{});
    return k;
}

// All layers of R rows at a time with every weight of the network in shared
// memory: forward, and for TRAIN the output gradients 2 (y - t) / (B O) and
// the data gradients of all layers behind it. The weights are copied once a
// block, a layer a group, the sums of a layer wait for its group only;
// forward and backward read the same copy (W[n][k] along k and along n). Rows
// are taken in turns of the grid, so a network's weights are read once per
// resident block. A tile at a time through registers (kForward, kBackward)
// paid an L2 round trip and a barrier per tile, 14 of them for the tuner's
// network: 12.3 + 9.6 us of 239 rows, here 11.4 (7,000 cycles for the copies,
// 2,000 a layer, bound by shared memory: see termSums). Two columns a thread
// in four warps measured the same, one latency after another.
template <int R, bool TRAIN>
__global__ void __launch_bounds__(256) kResident(NetView v, const float *__restrict__ X, const float *__restrict__ T,
                                                 int B, int D, float *yOut) {
    extern __shared__ __align__(16) float smem[];
    constexpr int H = R / 2;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int col = threadIdx.x % 128, half = threadIdx.x / 128;
    const int last = v.layers - 1, in = v.dimIn[0], out = v.dimOut[last];
    int total = 0;
    for (int l = 0; l < v.layers; ++l) {
        const int K = v.dimIn[l], N = v.dimOut[l], ld = weightStride(K);
        const float *w = v.w[l];
        float *sw = smem + total;
        if (K % 4 == 0 && ((size_t)w & 15) == 0) {
            for (int k = 4 * lane; k < K; k += 128)
                for (int m = warp; m < N; m += 64)
#pragma unroll
                    for (int n = m; n < m + 64; n += 8)
                        if (n < N) copy16(sw + n * ld + k, w + n * K + k, true);
        } else {
            for (int k = lane; k < K; k += 32)
                for (int m = warp; m < N; m += 64)
#pragma unroll
                    for (int n = m; n < m + 64; n += 8)
                        if (n < N) copy4(sw + n * ld + k, w + n * K + k, true);
        }
        for (int n = threadIdx.x; n < N; n += 256) copy4(sw + N * ld + n, v.b[l] + n, true);
        copyCommit();
        total += layerFloats(K, N);
    }
    float *sx = smem + total;
    const float scale = 2.f / (float)(B * out);
    bool first = true;
    for (int m0 = blockIdx.x * R; m0 < B; m0 += gridDim.x * R, first = false) {
        int cur = 0, base = 0;
        __syncthreads();  // the rows before are done with
        for (int i = threadIdx.x; i < R * in; i += 256) {
            const int r = i / in, k = i % in;
            sx[(size_t)r * D + k] = m0 + r < B ? X[(size_t)(m0 + r) * in + k] : 0.f;
        }
        for (int l = 0; l < v.layers; ++l, cur ^= 1) {
            const int K = v.dimIn[l], N = v.dimOut[l], ld = weightStride(K);
            const float *sw = smem + base, *x = sx + (size_t)(cur * R + half * H) * D;
            float *xn = sx + (size_t)((cur ^ 1) * R + half * H) * D;
            if (first) copyWait(last - l);
            __syncthreads();  // the layer's weights and rows
            for (int n = col; n < N; n += 128) {
                const float *wr = sw + n * ld;
                float acc[H];
#pragma unroll
                for (int i = 0; i < H; ++i) acc[i] = 0.f;
                const int k = termSums<H>(acc, x, D, K, [&](int k) { return *(const float4 *)(wr + k); });
                for (int j = k; j < K; ++j)
#pragma unroll
                    for (int i = 0; i < H; ++i) acc[i] = fmaf(x[i * D + j], wr[j], acc[i]);
                const float bias = sw[N * ld + n];
#pragma unroll
                for (int i = 0; i < H; ++i) {
                    const int row = m0 + half * H + i;
                    float s = acc[i] + bias;
                    if (l < last) s = fmaxf(s, 0.f);
                    xn[(size_t)i * D + n] = s;
                    if (row >= B) continue;
                    if (TRAIN) v.act[l][(size_t)row * N + n] = s;
                    else if (l == last) yOut[(size_t)row * N + n] = s;
                }
            }
            base += layerFloats(K, N);
        }
        if (!TRAIN) continue;
        __syncthreads();
        for (int i = threadIdx.x; i < R * out; i += 256) {
            const int r = i / out, n = i % out;
            const size_t o = (size_t)(m0 + r) * out + n;
            float d = 0.f;
            if (m0 + r < B) v.delta[last][o] = d = scale * (sx[(size_t)(cur * R + r) * D + n] - T[o]);
            sx[(size_t)((cur ^ 1) * R + r) * D + n] = d;
        }
        cur ^= 1;
        for (int l = last; l > 0; --l, cur ^= 1) {
            const int K = v.dimOut[l], N = v.dimIn[l], ld = weightStride(N);
            base -= layerFloats(N, K);
            const float *sw = smem + base, *x = sx + (size_t)(cur * R + half * H) * D;
            float *xn = sx + (size_t)((cur ^ 1) * R + half * H) * D;
            __syncthreads();
            for (int n = col; n < N; n += 128) {
                float acc[H], act[H];  // act: this thread's own stores of the forward pass
#pragma unroll
                for (int i = 0; i < H; ++i) {
                    const int row = m0 + half * H + i;
                    acc[i] = 0.f;
                    act[i] = row < B ? v.act[l - 1][(size_t)row * N + n] : 0.f;
                }
                const int k = termSums<H>(acc, x, D, K, [&](int k) {
                    const float *wk = sw + k * ld + n;
                    return make_float4(wk[0], wk[ld], wk[2 * ld], wk[3 * ld]);
                });
                for (int j = k; j < K; ++j)
#pragma unroll
                    for (int i = 0; i < H; ++i) acc[i] = fmaf(x[i * D + j], sw[j * ld + n], acc[i]);
#pragma unroll
                for (int i = 0; i < H; ++i) {
                    const int row = m0 + half * H + i;
                    const float s = row < B && act[i] > 0.f ? acc[i] : 0.f;
                    if (row < B) v.delta[l - 1][(size_t)row * N + n] = s;
                    xn[(size_t)i * D + n] = s;
                }
            }
        }
    }
}

// Weight and bias gradients of every layer, one tile of 4 NW outputs x 32 KW
// inputs of one layer a block (grid.x) over rows [chunk * rows, ...) (grid.y):
// dW[n][k] = sum of delta[m][n] x[m][k], db[n] = sum of delta[m][n], in order
// of m. One chunk writes the gradients, more write their own copies (part +
// chunk * stride). The block after the tiles reduces the loss as kMse does.
// A thread holds NW outputs of KW inputs, which take NW + KW shared-memory
// accesses a row (a value that the whole warp reads costs one too): 2 x 1
// where one chain of rows leaves the GPU idle and the longest block counts, 4
// x 2 for chunks of rows. Slices of 32 rows are copied three ahead. With host
// (pinned memory) the gradients and the loss are written there too: a copy
// behind the kernels cost 5 us a call.
constexpr int kGradSlice = 32, kGradStages = 4;
template <int NW, int KW>
__global__ void __launch_bounds__(128) kWeightGrad(NetView v, const float *__restrict__ X, const float *__restrict__ T,
                                                   int B, int rows, const float *gradBase, float *part, size_t stride,
                                                   float *loss, float *host) {
    constexpr int kGradN = 4 * NW, kGradK = 32 * KW;
    __shared__ __align__(16) float sd[kGradStages][kGradSlice][kGradN];
    __shared__ __align__(16) float sx[kGradStages][kGradSlice][kGradK];
    // Set up while the pass before ends. It does not let this grid start
    // earlier: blocks that wait crowd on the SMs that are free then and stay
    // there (239 rows 24.6 us for both, so 18.5).
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == gridDim.x - 1) {
        if (blockIdx.y) return;
        float *sum = &sx[0][0][0];
        const float *y = v.act[v.layers - 1];
        const int count = B * v.dimOut[v.layers - 1];
        float s[2] = {0.f, 0.f};
        for (int i = threadIdx.x; i < count; i += 256)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (i + 128 * j < count) {
                    const float d = y[i + 128 * j] - T[i + 128 * j];
                    s[j] = fmaf(d, d, s[j]);
                }
        sum[threadIdx.x] = s[0] + s[1];
        __syncthreads();
        for (int w = 64; w > 0; w >>= 1) {
            if (threadIdx.x < w) sum[threadIdx.x] += sum[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            *loss = sum[0] / (float)count;
            if (host) host[loss - gradBase] = sum[0] / (float)count;
        }
        return;
    }
    int l = 0, tile = blockIdx.x, tk = 0;
    for (;; ++l) {
        tk = (v.dimIn[l] + kGradK - 1) / kGradK;
        const int tiles = tk * ((v.dimOut[l] + kGradN - 1) / kGradN);
        if (tile < tiles) break;
        tile -= tiles;
    }
    const int N = v.dimOut[l], K = v.dimIn[l];
    const int n0 = (tile / tk) * kGradN, k0 = (tile % tk) * kGradK;
    const float *d = v.delta[l], *x = l == 0 ? X : v.act[l - 1];
    const int m0 = blockIdx.y * rows, m1 = min(B, m0 + rows);
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const bool wide = K % 4 == 0 && ((size_t)x & 15) == 0;
    auto load = [&](int m, int stage) {
        if (m < m1) {
            if (wide) {
#pragma unroll
                for (int i = 0; i < 2 * KW; ++i) {
                    const int e = threadIdx.x + 128 * i, q = e / (8 * KW), k = 4 * (e % (8 * KW));
                    const bool on = m + q < m1 && k0 + k < K;
                    copy16(&sx[stage][q][k], on ? x + (size_t)(m + q) * K + k0 + k : x, on);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8 * KW; ++i) {
                    const int e = threadIdx.x + 128 * i, q = e / kGradK, k = e % kGradK;
                    const bool on = m + q < m1 && k0 + k < K;
                    copy4(&sx[stage][q][k], on ? x + (size_t)(m + q) * K + k0 + k : x, on);
                }
            }
#pragma unroll
            for (int i = 0; i < NW; ++i) {
                const int e = threadIdx.x + 128 * i, q = e / kGradN, n = e % kGradN;
                const bool on = m + q < m1 && n0 + n < N;
                copy4(&sd[stage][q][n], on ? d + (size_t)(m + q) * N + n0 + n : d, on);
            }
        }
        copyCommit();
    };
    for (int i = 0; i < kGradStages - 1; ++i) load(m0 + i * kGradSlice, i);
    float acc[NW][KW] = {}, bias[NW] = {};
    int stage = 0;
    for (int m = m0; m < m1; m += kGradSlice, stage = (stage + 1) % kGradStages) {
        copyWait(kGradStages - 2);
        __syncthreads();  // this slice is there, and the one before is done with
        load(m + (kGradStages - 1) * kGradSlice, (stage + kGradStages - 1) % kGradStages);
        const int end = min(kGradSlice, m1 - m);
        auto step = [&](int q) {
            float dn[NW], xk[KW];
#pragma unroll
            for (int j = 0; j < NW; ++j) dn[j] = sd[stage][q][NW * warp + j];
#pragma unroll
            for (int j = 0; j < KW; ++j) xk[j] = sx[stage][q][32 * j + lane];
#pragma unroll
            for (int j = 0; j < NW; ++j) {
#pragma unroll
                for (int i = 0; i < KW; ++i) acc[j][i] = fmaf(dn[j], xk[i], acc[j][i]);
                bias[j] += dn[j];
            }
        };
        if (end == kGradSlice) {
#pragma unroll 16
            for (int q = 0; q < kGradSlice; ++q) step(q);
        } else {
            for (int q = 0; q < end; ++q) step(q);
        }
    }
    float *dw = v.dw[l], *db = v.db[l];
    if (part) {
        dw = part + (size_t)blockIdx.y * stride + (dw - gradBase);
        db = part + (size_t)blockIdx.y * stride + (db - gradBase);
    }
#pragma unroll
    for (int j = 0; j < NW; ++j) {
        const int n = n0 + NW * warp + j;
        if (n >= N) continue;
#pragma unroll
        for (int i = 0; i < KW; ++i) {
            const int k = k0 + 32 * i + lane;
            if (k >= K) continue;
            dw[(size_t)n * K + k] = acc[j][i];
            if (host && !part) host[dw - gradBase + (size_t)n * K + k] = acc[j][i];
        }
        if (k0 == 0 && lane == 0) {
            db[n] = bias[j];
            if (host && !part) host[db - gradBase + n] = bias[j];
        }
    }
}

// Sum of the chunks' gradients, in order of the chunks.
__global__ void __launch_bounds__(256) kGradReduce(long long n, int chunks, const float *__restrict__ part,
                                                   size_t stride, float *__restrict__ grad, float *host) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = part[i];
    for (int c = 1; c < chunks; ++c) s += part[c * stride + i];
    grad[i] = s;
    if (host) host[i] = s;
}

// Adam (Kingma & Ba 2015) with bias correction.
__global__ void kAdam(long long n, float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                      float *__restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

template <bool TA, bool TB>
void gemm(cudaStream_t s, int M, int N, int K, const float *A, int lda, const float *B, int ldb, float *C, int ldc,
          int epi, const float *bias, const float *mask) {
    dim3 grid(ceilDiv(N, kT), ceilDiv(M, kT));
    kGemm<TA, TB><<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, ldc, epi, bias, mask);
    RACE_CUDA(cudaGetLastError());
}

}  // namespace

struct Mlp {
    int in = 0, hidden = 0, hiddenLayers = 0, out = 0;
    std::vector<int> dimIn, dimOut;
    std::vector<size_t> wOff, bOff;
    size_t numParams = 0;
    DevBuf<float> params, grads, m1, m2;
    DevBuf<float> acts, deltas;  // activations per layer, gradients of them (one product at a time: two of the widest)
    DevBuf<float> part;          // gradients of chunks of rows
    float *hostGrads = nullptr;  // pinned: gradients and loss on their way to the caller
    bool fused = false;          // has passes of one kernel (else one kernel per product)
    unsigned sharedAllowed = 0;  // allowShared's kernels, a bit each
    int batchCap = 0;
    long long steps = 0;

    Mlp(int in_, int hidden_, int layers_, int out_) : in(in_), hidden(hidden_), hiddenLayers(layers_), out(out_) {
        if (in < 1 || hidden < 1 || layers_ < 1 || out < 1) throw Error(RACE_ERR_INVALID_ARG, "bad MLP shape");
        for (int l = 0; l <= hiddenLayers; ++l) {
            dimIn.push_back(l == 0 ? in : hidden);
            dimOut.push_back(l == hiddenLayers ? out : hidden);
            wOff.push_back(numParams);
            numParams += (size_t)dimIn.back() * dimOut.back();
            bOff.push_back(numParams);
            numParams += dimOut.back();
        }
        params.alloc(numParams);
        grads.alloc(numParams + 1);  // the loss follows the gradients
        m1.alloc(numParams);
        m2.alloc(numParams);
        fused = layers() <= kFusedLayers && std::max(in, std::max(hidden, out)) <= kFusedDim;
        RACE_CUDA(cudaMemset(params.p, 0, sizeof(float) * numParams));
        RACE_CUDA(cudaMemset(m1.p, 0, sizeof(float) * numParams));
        RACE_CUDA(cudaMemset(m2.p, 0, sizeof(float) * numParams));
    }
    Mlp(const Mlp &) = delete;
    Mlp &operator=(const Mlp &) = delete;
    ~Mlp() {
        if (hostGrads) cudaFreeHost(hostGrads);
    }
    float *loss() { return grads.p + numParams; }
    int layers() const { return hiddenLayers + 1; }
    // activation l (l = 1..layers) of a batch row: output of layer l-1
    size_t actOff(int l, int B) const {
        size_t o = 0;
        for (int i = 1; i < l; ++i) o += (size_t)B * dimOut[i - 1];
        return o;
    }
    // A batch is limited by the second grid dimension of kGemm; the fused
    // passes count rows and outputs in 32 bits within it.
    static void checkBatch(int B) {
        if (B > 65535 * kT) throw Error(RACE_ERR_INVALID_ARG, "a batch holds at most 2,097,120 rows");
    }
    void ensure(int B) {
        if (B <= batchCap) return;
        size_t total = 0, widest = 0;
        for (int l = 0; l < layers(); ++l) {
            total += (size_t)B * dimOut[l];
            widest = std::max(widest, (size_t)B * std::max(dimOut[l], dimIn[l]));
        }
        acts.alloc(total);
        deltas.alloc(fused ? std::max(total, 2 * widest) : 2 * widest);  // fused networks: both forms (byProducts)
        if (fused && gradChunks(B) > 1) part.ensure(gradStride() * gradChunks(B));
        batchCap = B;
    }
    // Rows that one chain of the fused weight gradients sums, and their chunks:
    // one chain per gradient up to kGradRows rows; above, chunks of rows fill
    // the GPU (168 small tiles of the tuner's network fill it once, 42 large
    // ones do not). More rows never mean fewer chunks, so the workspace of a
    // batch serves every smaller one.
    static int gradRows(int B) { return B <= kGradRows ? B : std::max(kGradChunk, ceilDiv(B, kGradChunks)); }
    static int gradChunks(int B) { return ceilDiv(B, gradRows(B)); }
    size_t gradStride() const { return (numParams + 31) & ~(size_t)31; }
    NetView view(int B) const {
        NetView v{};
        v.layers = layers();
        for (int l = 0; l < layers(); ++l) {
            v.dimIn[l] = dimIn[l];
            v.dimOut[l] = dimOut[l];
            v.w[l] = params.p + wOff[l];
            v.b[l] = params.p + bOff[l];
            v.dw[l] = grads.p + wOff[l];
            v.db[l] = grads.p + bOff[l];
            if (B > 0) {
                v.act[l] = acts.p + actOff(l + 1, B);
                v.delta[l] = deltas.p + actOff(l + 1, B);
            }
        }
        return v;
    }
    // shared memory of R rows of two layers, the widest padded to whole float4
    int rowStride() const { return (std::max(in, std::max(hidden, out)) + 3) & ~3; }
    static int passBytes(int R, int stride) { return (int)(kTileBytes + 2 * R * stride * sizeof(float)); }
    // Rows a block: 2 while that leaves at most one block an SM (239 rows: 120
    // blocks, 18.5 us for loss and gradients, 4 rows 20.5), then 4 and 8, and 16
    // where enough blocks remain to share each weight among more rows.
    static int rowsPerBlock(int B) { return B <= 2 * 152 ? 2 : B <= 4 * 152 ? 4 : B <= 8 * 152 ? 8 : 16; }
    // Lets a kernel take more than 48 KB of shared memory. That holds for one
    // device, the network's own, so each network asks once per kernel (slot).
    static int rowsIndex(int R) { return R == 2 ? 0 : R == 4 ? 1 : R == 8 ? 2 : 3; }
    template <typename K>
    void allowShared(K kernel, int slot, int bytes) {
        if (sharedAllowed >> slot & 1) return;
        RACE_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        sharedAllowed |= 1u << slot;
    }
    template <int R>
    void fusedForward(const NetView &v, const float *X, int B, float *y, cudaStream_t s) {
        allowShared(kForward<R>, 0 + rowsIndex(R), passBytes(R, kFusedDim));
        kForward<R><<<ceilDiv(B, R), 256, passBytes(R, rowStride()), s>>>(v, X, B, rowStride(), y);
    }
    template <int R>
    void fusedBackward(const NetView &v, const float *T, int B, cudaStream_t s) {
        allowShared(kBackward<R>, 4 + rowsIndex(R), passBytes(R, kFusedDim));
        kBackward<R><<<ceilDiv(B, R), 256, passBytes(R, rowStride()), s>>>(v, T, B, rowStride());
    }
    // Shared memory of the whole network and R rows of two layers (164 KB for
    // the tuner's network and 8 rows); where it fits, kResident takes the pass
    // (239 rows, loss and gradients on the GPU: 33 us by tiles, 18.5 resident).
    size_t residentBytes(int R) const {
        size_t f = 2 * (size_t)R * rowStride();
        for (int l = 0; l < layers(); ++l) f += layerFloats(dimIn[l], dimOut[l]);
        return sizeof(float) * f;
    }
    template <int R, bool TRAIN>
    bool residentPass(const NetView &v, const float *X, const float *T, int B, float *y, cudaStream_t s) {
        const size_t bytes = residentBytes(R);
        if (bytes > kResidentBytes) return false;
        allowShared(kResident<R, TRAIN>, (TRAIN ? 12 : 8) + rowsIndex(R), (int)kResidentBytes);
        const int perSm = (int)std::max<size_t>(1, std::min<size_t>(8, kResidentBytes / (bytes + 1024)));
        kResident<R, TRAIN><<<std::min(ceilDiv(B, R), kResidentSms * perSm), 256, bytes, s>>>(v, X, T, B, rowStride(), y);
        return true;
    }
    template <typename F>
    void byRows(int B, F &&f) {
        switch (rowsPerBlock(B)) {
        case 16: f(std::integral_constant<int, 16>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        default: f(std::integral_constant<int, 2>{}); break;
        }
        RACE_CUDA(cudaGetLastError());
    }
    static bool capturing(cudaStream_t s) {
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        RACE_CUDA(cudaStreamIsCapturing(s, &st));
        return st != cudaStreamCaptureStatusNone;
    }
    // Whether a batch runs one kernel per product: networks that no fused pass
    // takes, and wide ones with few rows. A fused block of a few rows goes
    // through all weights by itself, 1.2 us a tile; a product's blocks share
    // them and take 0.083 us a term of their sums (0.072 up to one row of
    // blocks, 1.2 times that where they do not fit on the GPU at once).
    // Measured, outputs and gradients, fused / by products, microseconds:
    // 34-1024-1024-1024-1, 64 rows 341 and 701 / 255 and 469, 256 rows 342 and
    // 762 / 309 and 658, 320 rows 389 and 870 / 412 and 866; 34-768-768-768-1,
    // 16 rows 197 and 395 / 173 and 314, 256 rows 200 and 441 / 239 and 512;
    // 34-512-512-512-1, 64 rows 97 and 193 / 136 and 263.
    bool byProducts(int B) const {
        if (!fused) return true;
        if (B > 256 || residentBytes(rowsPerBlock(B)) <= kResidentBytes) return false;
        long long tiles = 0, terms = 0, blocks = 0;
        for (int l = 0; l < layers(); ++l) {
            tiles += (long long)ceilDiv(dimOut[l], kTileN) * ceilDiv(dimIn[l], kTileK);
            terms += dimIn[l];
            blocks = std::max(blocks, (long long)ceilDiv(dimOut[l], kT) * ceilDiv(B, kT));
        }
        return (B <= kT ? 0.072 : 0.083) * terms * (blocks > kResidentSms ? 1.2 : 1.0) < 1.2 * tiles;
    }
    // outputs only, to Y
    void predict(const float *X, int B, float *Y, cudaStream_t s) {
        // (a capture cannot allocate the products' workspace; the fused pass needs none)
        if (!fused || (byProducts(B) && (B <= batchCap || !capturing(s)))) {
            const float *y = forward(X, B, s);
            RACE_CUDA(cudaMemcpyAsync(Y, y, sizeof(float) * B * out, cudaMemcpyDeviceToDevice, s));
            return;
        }
        // Outputs alone need no workspace, but the first pass of a batch size
        // is also a later captured training pass's chance to allocate.
        if (B > batchCap && !capturing(s)) ensure(B);
        // Blocks write outputs while others still read inputs: outputs that
        // share memory with the inputs are put together apart from them.
        const bool overlap = Y < X + (size_t)B * in && X < Y + (size_t)B * out;
        if (overlap) ensure(B);
        float *y = overlap ? acts.p + actOff(layers(), B) : Y;
        const NetView v = view(0);
        byRows(B, [&](auto r) {
            constexpr int R = decltype(r)::value;
            if (!residentPass<R, false>(v, X, nullptr, B, y, s)) fusedForward<R>(v, X, B, y, s);
        });
        if (overlap) RACE_CUDA(cudaMemcpyAsync(Y, y, sizeof(float) * B * out, cudaMemcpyDeviceToDevice, s));
    }
    template <int NW, int KW>
    void weightGrad(const NetView &v, const float *X, const float *T, int B, int rows, int chunks, size_t stride,
                    float *host, cudaStream_t s) {
        int tiles = 0;
        for (int l = 0; l < layers(); ++l) tiles += ceilDiv(dimOut[l], 4 * NW) * ceilDiv(dimIn[l], 32 * KW);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(tiles + 1, chunks);
        cfg.blockDim = dim3(128);
        cfg.stream = s;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeProgrammaticStreamSerialization;  // starts as the pass ends, waits for it
        at.val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        RACE_CUDA(cudaLaunchKernelEx(&cfg, kWeightGrad<NW, KW>, v, X, T, B, rows, (const float *)grads.p,
                                     chunks > 1 ? part.p : (float *)nullptr, stride, loss(), host));
    }
    void lossGradFused(const float *X, const float *T, int B, float *host, cudaStream_t s) {
        ensure(B);
        const NetView v = view(B);
        byRows(B, [&](auto r) {
            constexpr int R = decltype(r)::value;
            if (residentPass<R, true>(v, X, T, B, nullptr, s)) return;
            fusedForward<R>(v, X, B, nullptr, s);
            fusedBackward<R>(v, T, B, s);
        });
        const int rows = gradRows(B), chunks = gradChunks(B);
        const size_t stride = gradStride();
        if (chunks == 1) weightGrad<2, 1>(v, X, T, B, rows, chunks, stride, host, s);
        else weightGrad<4, 2>(v, X, T, B, rows, chunks, stride, host, s);
        if (chunks > 1) {
            kGradReduce<<<ceilDiv((long long)numParams, 256), 256, 0, s>>>((long long)numParams, chunks, part.p, stride,
                                                                          grads.p, host);
            RACE_CUDA(cudaGetLastError());
        }
    }
    // forward: activations of every layer into acts; returns the output pointer
    float *forward(const float *X, int B, cudaStream_t s) {
        ensure(B);
        const float *x = X;
        for (int l = 0; l < layers(); ++l) {
            float *y = acts.p + actOff(l + 1, B);
            const bool last = l == layers() - 1;
            gemm<false, true>(s, B, dimOut[l], dimIn[l], x, dimIn[l], params.p + wOff[l], dimIn[l], y, dimOut[l],
                              last ? EPI_BIAS : EPI_BIAS_RELU, params.p + bOff[l], nullptr);
            x = y;
        }
        return acts.p + actOff(layers(), B);
    }
    // loss and gradients of the MSE against targets T (B x out); returns
    // whether the kernels wrote them to host too
    bool lossGrad(const float *X, const float *T, int B, float *host, cudaStream_t s) {
        if (!byProducts(B)) {
            lossGradFused(X, T, B, host, s);
            return host != nullptr;
        }
        float *y = forward(X, B, s);
        float *d = deltas.p, *dNext = deltas.p + deltas.n / 2;
        kMse<<<1, 256, 0, s>>>(B * out, y, T, d, loss());
        RACE_CUDA(cudaGetLastError());
        for (int l = layers() - 1; l >= 0; --l) {
            const float *xin = l == 0 ? X : acts.p + actOff(l, B);
            // dW = d^T xin  [out_l x in_l], db = column sums of d
            gemm<true, false>(s, dimOut[l], dimIn[l], B, d, dimOut[l], xin, dimIn[l], grads.p + wOff[l], dimIn[l],
                              EPI_NONE, nullptr, nullptr);
            kColSum<<<ceilDiv(dimOut[l], 128), 128, 0, s>>>(B, dimOut[l], d, grads.p + bOff[l]);
            RACE_CUDA(cudaGetLastError());
            if (l > 0) {
                // d_prev = (d W) * (xin > 0): xin is the ReLU output of layer l-1
                gemm<false, false>(s, B, dimIn[l], dimOut[l], d, dimOut[l], params.p + wOff[l], dimIn[l], dNext,
                                   dimIn[l], EPI_RELU_MASK, nullptr, xin);
                std::swap(d, dNext);
            }
        }
        return false;
    }
    void adam(float lr, float b1, float b2, float eps, cudaStream_t s) {
        ++steps;
        const float c1 = 1.f - std::pow(b1, (float)steps), c2 = 1.f - std::pow(b2, (float)steps);
        kAdam<<<ceilDiv((long long)numParams, 256), 256, 0, s>>>((long long)numParams, params.p, grads.p, m1.p, m2.p,
                                                                lr, b1, b2, eps, c1, c2);
        RACE_CUDA(cudaGetLastError());
    }
};

}  // namespace race

struct race_mlp {
    std::unique_ptr<race::Mlp> net;
    std::string err;
};

namespace {
template <typename F>
int guardMlp(race_mlp *h, F &&f) {
    try {
        f();
        return RACE_SUCCESS;
    } catch (const race::Error &ex) {
        if (h) h->err = ex.what();
        return ex.code;
    } catch (const std::exception &ex) {
        if (h) h->err = ex.what();
        return RACE_ERR_INTERNAL;
    }
}
}  // namespace

extern "C" {

int race_mlp_create(race_mlp **out, int in, int hidden, int hiddenLayers, int outDim) {
    if (!out) return RACE_ERR_INVALID_ARG;
    *out = nullptr;
    race_mlp *h = new race_mlp;
    int rc = guardMlp(h, [&] { h->net = std::make_unique<race::Mlp>(in, hidden, hiddenLayers, outDim); });
    if (rc != RACE_SUCCESS) {
        delete h;
        return rc;
    }
    *out = h;
    return RACE_SUCCESS;
}

int race_mlp_destroy(race_mlp *h) {
    delete h;
    return RACE_SUCCESS;
}

int race_mlp_num_params(race_mlp *h, long long *count) {
    if (!h || !count) return RACE_ERR_INVALID_ARG;
    *count = (long long)h->net->numParams;
    return RACE_SUCCESS;
}

int race_mlp_set_params(race_mlp *h, const float *host, long long count) {
    if (!h || !host || count != (long long)h->net->numParams) return RACE_ERR_INVALID_ARG;
    return guardMlp(h, [&] {
        RACE_CUDA(cudaMemcpy(h->net->params.p, host, sizeof(float) * count, cudaMemcpyHostToDevice));
        RACE_CUDA(cudaMemset(h->net->m1.p, 0, sizeof(float) * count));
        RACE_CUDA(cudaMemset(h->net->m2.p, 0, sizeof(float) * count));
        h->net->steps = 0;
    });
}

int race_mlp_get_params(race_mlp *h, float *host, long long count) {
    if (!h || !host || count != (long long)h->net->numParams) return RACE_ERR_INVALID_ARG;
    return guardMlp(h, [&] {
        RACE_CUDA(cudaMemcpy(host, h->net->params.p, sizeof(float) * count, cudaMemcpyDeviceToHost));
    });
}

int race_mlp_forward(race_mlp *h, const float *X, int batch, float *Y, void *stream) {
    if (!h || !X || !Y || batch < 1) return RACE_ERR_INVALID_ARG;
    return guardMlp(h, [&] {
        race::Mlp::checkBatch(batch);
        h->net->predict(X, batch, Y, (cudaStream_t)stream);
    });
}

int race_mlp_loss_grad(race_mlp *h, const float *X, const float *T, int batch, float *loss_host, float *grad_host,
                       void *stream) {
    if (!h || !X || !T || batch < 1) return RACE_ERR_INVALID_ARG;
    return guardMlp(h, [&] {
        cudaStream_t s = (cudaStream_t)stream;
        // The kernels write what the caller wants to pinned memory themselves
        // (52 -> 47 us a call of 239 rows); one product at a time copies it.
        race::Mlp &net = *h->net;
        race::Mlp::checkBatch(batch);
        const bool wanted = loss_host || grad_host;
        if (wanted && !net.hostGrads)
            RACE_CUDA(cudaMallocHost((void **)&net.hostGrads, sizeof(float) * (net.numParams + 1)));
        const bool there = net.lossGrad(X, T, batch, grad_host ? net.hostGrads : nullptr, s);
        if (!wanted) return;
        if (!there) {
            const size_t first = grad_host ? 0 : net.numParams;
            RACE_CUDA(cudaMemcpyAsync(net.hostGrads + first, net.grads.p + first,
                                      sizeof(float) * (net.numParams + 1 - first), cudaMemcpyDeviceToHost, s));
        }
        RACE_CUDA(cudaStreamSynchronize(s));
        if (grad_host) std::memcpy(grad_host, net.hostGrads, sizeof(float) * net.numParams);
        if (loss_host) *loss_host = net.hostGrads[net.numParams];
    });
}

int race_mlp_adam_step(race_mlp *h, float lr, float beta1, float beta2, float eps, void *stream) {
    if (!h || !(lr > 0.f)) return RACE_ERR_INVALID_ARG;
    return guardMlp(h, [&] { h->net->adam(lr, beta1, beta2, eps, (cudaStream_t)stream); });
}

const char *race_mlp_last_error(race_mlp *h) { return h ? h->err.c_str() : "null network"; }

}  // extern "C"
