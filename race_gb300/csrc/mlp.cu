// Multilayer perceptron of the parameter tuner: forward pass, mean-squared-
// error gradients and Adam updates as hand-written CUDA kernels (FP32).
//
// Network: in -> hidden (ReLU) -> ... (hiddenLayers times) -> out, every
// layer y = x W^T + b with W stored row-major [outDim][inDim]. Parameters
// are one flat array: for each layer W then b. The tuner's network is small
// (34 inputs, 3 x 128 hidden, 1 output) and its batches are some hundreds to
// thousands of rows: a product is a few million multiply-adds, so launches and
// the latency of each bound the time, not arithmetic. The whole forward pass
// is therefore one kernel (kForward: a block takes a few rows through all
// layers, activations in shared memory, weights in tiles fetched one ahead
// across the layer boundaries), the loss and the data gradients another
// (kBackward) and all layers' weight and bias gradients a third (kWeightGrad).
// One kernel per product took 16 launches: loss and gradients of 239 rows
// were 146 us on the GPU (222 us a call), one 32 x 32 tile after another for
// the weight gradients and one thread per column for the bias sums; now 32 us
// in three launches (77 us a call, the rest is the gradients' way to the
// caller's host memory).
// Networks wider than kFusedDim or deeper than kFusedLayers run the products
// one by one (kGemm: 32 x 32 output tiles, 16-deep k slices).
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
// for R rows; block 0 also reduces the loss as kMse does.
template <int R>
__global__ void __launch_bounds__(256) kBackward(NetView v, const float *__restrict__ T, int B, int D, float *loss) {
    extern __shared__ __align__(16) float smem[];
    auto sw = (float(*)[kTileK][kTileN + 1]) smem;
    float *sx = smem + kTileBytes / sizeof(float);
    const int m0 = blockIdx.x * R, last = v.layers - 1, out = v.dimOut[last], count = B * out;
    const float *y = v.act[last];
    const float scale = 2.f / (float)count;
    if (blockIdx.x == 0) {
        __shared__ float part[256];
        float s = 0.f;
        for (int i = threadIdx.x; i < count; i += 256) {
            const float d = y[i] - T[i];
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

// Weight and bias gradients of every layer, one 32 x 32 tile of one layer a
// block (grid.x) over rows [chunk * rows, ...) (grid.y): dW[n][k] = sum of
// delta[m][n] x[m][k], db[n] = sum of delta[m][n], in order of m. One chunk
// writes the gradients, more write their own copies (part + chunk * stride).
constexpr int kGradTile = 32, kGradSlice = 32;
__global__ void __launch_bounds__(256) kWeightGrad(NetView v, const float *__restrict__ X, int B, int rows,
                                                   const float *gradBase, float *part, size_t stride) {
    __shared__ float sd[2][kGradSlice][kGradTile + 1], sx[2][kGradSlice][kGradTile + 1];
    int l = 0, tile = blockIdx.x, tk = 0;
    for (;; ++l) {
        tk = (v.dimIn[l] + kGradTile - 1) / kGradTile;
        const int tiles = tk * ((v.dimOut[l] + kGradTile - 1) / kGradTile);
        if (tile < tiles) break;
        tile -= tiles;
    }
    const int N = v.dimOut[l], K = v.dimIn[l];
    const int n0 = (tile / tk) * kGradTile, k0 = (tile % tk) * kGradTile;
    const float *d = v.delta[l], *x = l == 0 ? X : v.act[l - 1];
    const int m0 = blockIdx.y * rows, m1 = min(B, m0 + rows);
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float rd[4], rx[4], acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, bias = 0.f;
    auto load = [&](int m) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = m + warp + 8 * i;
            rd[i] = row < m1 && n0 + lane < N ? d[(size_t)row * N + n0 + lane] : 0.f;
            rx[i] = row < m1 && k0 + lane < K ? x[(size_t)row * K + k0 + lane] : 0.f;
        }
    };
    load(m0);
    int buf = 0;
    for (int m = m0; m < m1; m += kGradSlice, buf ^= 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            sd[buf][warp + 8 * i][lane] = rd[i];
            sx[buf][warp + 8 * i][lane] = rx[i];
        }
        __syncthreads();
        if (m + kGradSlice < m1) load(m + kGradSlice);
        const int end = min(kGradSlice, m1 - m);
#pragma unroll 8
        for (int q = 0; q < end; ++q) {
            const float d0 = sd[buf][q][ty], d1 = sd[buf][q][ty + 16], x0 = sx[buf][q][tx], x1 = sx[buf][q][tx + 16];
            acc[0][0] = fmaf(d0, x0, acc[0][0]);
            acc[0][1] = fmaf(d0, x1, acc[0][1]);
            acc[1][0] = fmaf(d1, x0, acc[1][0]);
            acc[1][1] = fmaf(d1, x1, acc[1][1]);
        }
        if (k0 == 0 && warp == 0)
            for (int q = 0; q < end; ++q) bias += sd[buf][q][lane];
    }
    float *dw = v.dw[l], *db = v.db[l];
    if (part) {
        dw = part + (size_t)blockIdx.y * stride + (dw - gradBase);
        db = part + (size_t)blockIdx.y * stride + (db - gradBase);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int n = n0 + ty + 16 * i, k = k0 + tx + 16 * j;
            if (n < N && k < K) dw[(size_t)n * K + k] = acc[i][j];
        }
    if (k0 == 0 && warp == 0 && n0 + lane < N) db[n0 + lane] = bias;
}

// Sum of the chunks' gradients, in order of the chunks.
__global__ void __launch_bounds__(256) kGradReduce(long long n, int chunks, const float *__restrict__ part,
                                                   size_t stride, float *__restrict__ grad) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = part[i];
    for (int c = 1; c < chunks; ++c) s += part[c * stride + i];
    grad[i] = s;
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
    bool fused = false;          // one kernel per pass (else one per product)
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
    void ensure(int B) {
        if (B <= batchCap) return;
        size_t total = 0, widest = 0;
        for (int l = 0; l < layers(); ++l) {
            total += (size_t)B * dimOut[l];
            widest = std::max(widest, (size_t)B * std::max(dimOut[l], dimIn[l]));
        }
        acts.alloc(total);
        deltas.alloc(fused ? total : 2 * widest);
        batchCap = B;
    }
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
    // Rows a block: 4 while that leaves at most one block an SM (239 rows: 60
    // blocks), then 8, and 16 where enough blocks remain to share each weight
    // tile among more rows.
    static int rowsPerBlock(int B) { return B <= 4 * 152 ? 4 : B <= 8 * 152 ? 8 : 16; }
    template <int R>
    void fusedForward(const NetView &v, const float *X, int B, float *y, cudaStream_t s) {
        static const cudaError_t opt = cudaFuncSetAttribute(
            kForward<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, passBytes(R, kFusedDim));
        RACE_CUDA(opt);
        kForward<R><<<ceilDiv(B, R), 256, passBytes(R, rowStride()), s>>>(v, X, B, rowStride(), y);
    }
    template <int R>
    void fusedBackward(const NetView &v, const float *T, int B, cudaStream_t s) {
        static const cudaError_t opt = cudaFuncSetAttribute(
            kBackward<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, passBytes(R, kFusedDim));
        RACE_CUDA(opt);
        kBackward<R><<<ceilDiv(B, R), 256, passBytes(R, rowStride()), s>>>(v, T, B, rowStride(), loss());
    }
    template <typename F>
    void byRows(int B, F &&f) {
        switch (rowsPerBlock(B)) {
        case 16: f(std::integral_constant<int, 16>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        default: f(std::integral_constant<int, 4>{}); break;
        }
        RACE_CUDA(cudaGetLastError());
    }
    // outputs only, to Y
    void predict(const float *X, int B, float *Y, cudaStream_t s) {
        if (!fused) {
            const float *y = forward(X, B, s);
            RACE_CUDA(cudaMemcpyAsync(Y, y, sizeof(float) * B * out, cudaMemcpyDeviceToDevice, s));
            return;
        }
        const NetView v = view(0);
        byRows(B, [&](auto r) { fusedForward<decltype(r)::value>(v, X, B, Y, s); });
    }
    void lossGradFused(const float *X, const float *T, int B, cudaStream_t s) {
        ensure(B);
        const NetView v = view(B);
        byRows(B, [&](auto r) { fusedForward<decltype(r)::value>(v, X, B, nullptr, s); });
        byRows(B, [&](auto r) { fusedBackward<decltype(r)::value>(v, T, B, s); });
        int tiles = 0;
        for (int l = 0; l < layers(); ++l) tiles += ceilDiv(dimOut[l], kGradTile) * ceilDiv(dimIn[l], kGradTile);
        // one chain per gradient up to kGradRows rows; above, chunks of rows
        // fill the GPU (44 tiles of the tuner's network leave 108 SMs idle)
        const int rows = B <= kGradRows ? B : std::max(kGradChunk, ceilDiv(B, kGradChunks));
        const int chunks = ceilDiv(B, rows);
        const size_t stride = (numParams + 31) & ~(size_t)31;
        if (chunks > 1) part.ensure(stride * chunks);
        kWeightGrad<<<dim3(tiles, chunks), 256, 0, s>>>(v, X, B, rows, grads.p, chunks > 1 ? part.p : nullptr, stride);
        RACE_CUDA(cudaGetLastError());
        if (chunks > 1) {
            kGradReduce<<<ceilDiv((long long)numParams, 256), 256, 0, s>>>((long long)numParams, chunks, part.p, stride,
                                                                          grads.p);
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
    // loss and gradients of the MSE against targets T (B x out)
    void lossGrad(const float *X, const float *T, int B, cudaStream_t s) {
        if (fused) return lossGradFused(X, T, B, s);
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
        h->net->predict(X, batch, Y, (cudaStream_t)stream);
    });
}

int race_mlp_loss_grad(race_mlp *h, const float *X, const float *T, int batch, float *loss_host, float *grad_host,
                       void *stream) {
    if (!h || !X || !T || batch < 1) return RACE_ERR_INVALID_ARG;
    return guardMlp(h, [&] {
        cudaStream_t s = (cudaStream_t)stream;
        h->net->lossGrad(X, T, batch, s);
        if (!loss_host && !grad_host) return;
        // one copy through pinned memory (a pageable copy waits by itself,
        // and there were two)
        race::Mlp &net = *h->net;
        if (!net.hostGrads) RACE_CUDA(cudaMallocHost((void **)&net.hostGrads, sizeof(float) * (net.numParams + 1)));
        const size_t first = grad_host ? 0 : net.numParams;
        RACE_CUDA(cudaMemcpyAsync(net.hostGrads + first, net.grads.p + first, sizeof(float) * (net.numParams + 1 - first),
                                  cudaMemcpyDeviceToHost, s));
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
