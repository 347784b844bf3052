// Gather execution (RACE_SWEEP_GATHER) of SpMV, SpMTV and SymmSpMV: one
// thread per entry of b, which replays the updates RACE's sequential walk
// makes to it, in that walk's order (GatherPlan, waves.h), with the kernel
// bodies' own operations (examples/src/helpers/kernels.cpp:5-15, 107-115,
// 403-417), so the results equal the wave executor's bit for bit; no phases,
// no grid barriers. SpMV has no updates of other rows: its thread sums its own
// row.
//
// Layout (large matrices with short rows have none: gatherPlain). The lists are
// per 32 consecutive entries of b (a warp) in groups of four updates per lane,
// so that a warp reads 512 contiguous bytes of matrix positions and of source
// rows at a time. The matrix values are always the
// caller's, in place (they may change between calls). A row's own SymmSpMV
// update (its diagonal, then its off-diagonal sum) stands in the list as its
// diagonal's position with the sign bit, so that every step is the same fma.
// Entries of b with many updates, or whose own row is long (foldLine), are
// folded by a warp each: it gathers 32 per lane and round while all lanes
// run the chain.
//
// What bounds it on GB300: the FP64 pipe (2 fma a cycle and SM: 32 us for the
// 10.4M stored entries of the 27-point 95x87x91 SymmSpMV) and the L1 (one
// 32-byte sector per lane for the values of other rows' updates and for the
// own row); for long entries the chain of a fold (FP64: 64 cycles an update).
// Measured, b zeroed and one call, before (a thread per entry of b on the
// caller's CRS and plain lists) and now: SymmSpMV FP64 27-point 95x87x91 124
// and 90 us, 7-point 32^3 14.6 and 10.2 us; SpMTV FP64 27-point 80x81x79 167
// and 60 us; SpMV there 50.0 and 45.5 us; on a 60k-row power-law graph (lists
// of up to 20k updates) SymmSpMV FP64 4,184 and 1,589 us, FP32 2,281 and 313
// us, SpMTV FP32 8,855 and 666 us.
#include <algorithm>
#include <climits>
#include <utility>

#include "engine.h"
#include "sweep_ops.cuh"

namespace race {
namespace {

constexpr int kGatherThreads = 128;
constexpr int kGatherWarps = kGatherThreads / 32;
// Least number of updates of an entry that a warp gathers for (foldLine): a
// thread's chain of that many takes as long as the rest of a small launch
// (lists of a stencil stay below: 26).
constexpr int kLongList = 96;

struct GatherArgs {
    int n, numLong;
    const int *rowPtr, *col;
    const void *val, *x;
    void *b;
    const int *len;  // per entry of b: updates in its list (-1: a long one)
    const long long *listOff;           // per chunk of 32 entries of b
    const int *listPos, *listSrc;       // matrix position (sign bit: the row's own update) and source row
    const int *longY, *ptr, *entry, *src;  // the long ones: GatherPlan's lists
};

// Entries [0, cnt) of a fold, f(k) their (value, x) pair, applied in order to
// acc by every lane: each lane gathers P of them a round, the next round's
// in flight while this one's are applied.
template <typename XT>
struct Pair {
    XT v, x;
    bool own;
};
template <typename XT, typename F, typename G>
__device__ __forceinline__ void warpFold(XT *sv, XT *sx, unsigned char *so, int cnt, int lane, F &&f, G &&apply) {
    constexpr int P = 4;
    Pair<XT> q[P];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int k = k0 + 32 * i + lane;
            q[i] = k < cnt ? f(k) : Pair<XT>{XT(0), XT(0), false};
        }
    };
    fetch(0);
    for (int k0 = 0; k0 < cnt; k0 += 32 * P) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < P; ++i) {
            sv[32 * i + lane] = q[i].v;
            sx[32 * i + lane] = q[i].x;
            so[32 * i + lane] = q[i].own;
        }
        __syncwarp();
        if (k0 + 32 * P < cnt) fetch(k0 + 32 * P);
        const int m = min(32 * P, cnt - k0);
#pragma unroll 8
        for (int i = 0; i < m; ++i) apply(sv[i], sx[i], so[i] != 0);
    }
}

// The long entries of b, a warp each. It lets the other entries' kernel start
// at once (programmatic dependent launch): both read x and write their own
// entries of b.
template <typename VT, typename XT, int KER>
__global__ void __launch_bounds__(kGatherThreads) kGatherLong(GatherArgs a) {
    constexpr bool kOwn = KER != RACE_K_SPMTV, kList = KER != RACE_K_SPMV, kSymm = KER == RACE_K_SYMMSPMV;
    __shared__ XT foldV[kGatherWarps][128], foldX[kGatherWarps][128];
    __shared__ unsigned char foldO[kGatherWarps][128];
    asm volatile("griddepcontrol.launch_dependents;");
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * kGatherWarps + w;
    if (i >= a.numLong) return;
    const VT *val = (const VT *)a.val;
    const XT *x = (const XT *)a.x;
    XT *b = (XT *)a.b;
    XT *sv = foldV[w], *sx = foldX[w];
    unsigned char *so = foldO[w];
    const int y = a.longY[i], s = a.rowPtr[y], e = a.rowPtr[y + 1];
    XT t = XT(0);
    if constexpr (kOwn) {
        const int j0 = s + (kSymm ? 1 : 0);
        warpFold<XT>(
            sv, sx, so, e - j0, lane,
            [&](int k) { return Pair<XT>{ld<VT, XT>(val, j0 + k), x[a.col[j0 + k]], false}; },
            [&](XT v, XT xv, bool) { t = mac(v, xv, t); });
    }
    XT acc = t;
    if constexpr (kList) {
        acc = b[y];
        const int k0 = a.ptr[y];
        warpFold<XT>(
            sv, sx, so, a.ptr[y + 1] - k0, lane,
            [&](int k) {
                const int p = a.entry[k0 + k];
                if (p >= 0) return Pair<XT>{ld<VT, XT>(val, p), x[a.src[k0 + k]], false};
                // the row's own update; a row without entries has none (adding -0
                // keeps a -0 as well)
                return e > s ? Pair<XT>{ld<VT, XT>(val, s), x[y], true} : Pair<XT>{XT(-0.0), XT(0), false};
            },
            [&](XT v, XT xv, bool own) {
                acc = mac(v, xv, acc);
                if (kSymm && own) acc += t;
            });
    }
    if (lane == 0) b[y] = acc;
}

// The other entries of b, a thread each. No shared memory: the L1 holds the
// sectors that neighbouring threads' CRS rows share.
// The own row's entries are taken eight at a time: columns, values, x, chain.
// The bound on resident blocks (8 of 128 threads: 64 registers) lets the
// compiler keep such a batch in flight; unbounded it took 32 registers for
// SpMV and spread the loads over the chain: 59 us instead of 49.5 us for the
// 27-point 80x81x79 in FP64, although twice as many threads were resident.
constexpr int kOwnBatch = 8;
constexpr int kShortThreads = 128, kShortBlocks = 8;
template <typename VT, typename XT, int KER>
__global__ void __launch_bounds__(kShortThreads, kShortBlocks)
    kGather(int n, int numLong, const int *__restrict__ rowPtr, const int *__restrict__ col, const VT *__restrict__ val,
            const XT *__restrict__ x, XT *__restrict__ b, const int *__restrict__ len,
            const long long *__restrict__ listOff, const int *__restrict__ listPos, const int *__restrict__ listSrc) {
    constexpr bool kOwn = KER != RACE_K_SPMTV, kList = KER != RACE_K_SPMV, kSymm = KER == RACE_K_SYMMSPMV;
    const int y = blockIdx.x * kShortThreads + threadIdx.x, lane = threadIdx.x & 31;
    const int cnt = y < n ? (kList || numLong ? len[y] : 0) : -1;
    if (cnt >= 0) {
        XT t = XT(0);
        if constexpr (kOwn) {
            // eight entries' columns and values at once: a row's 32-byte
            // sectors are used up before other rows push them out of the L1
            constexpr int P = kOwnBatch;
            const int e = rowPtr[y + 1];
            int j = rowPtr[y] + (kSymm ? 1 : 0);
            for (; j + P <= e; j += P) {
                int c[P];
                XT v[P], xv[P];
#pragma unroll
                for (int k = 0; k < P; ++k) c[k] = col[j + k];
#pragma unroll
                for (int k = 0; k < P; ++k) v[k] = ld<VT, XT>(val, j + k);
#pragma unroll
                for (int k = 0; k < P; ++k) xv[k] = x[c[k]];
#pragma unroll
                for (int k = 0; k < P; ++k) t = mac(v[k], xv[k], t);
            }
            for (; j < e; ++j) t = mac(ld<VT, XT>(val, j), x[col[j]], t);
        }
        if constexpr (!kList) {
            b[y] = t;
        } else {
            const long long o = listOff[y >> 5] + 4 * lane;
            const int *pos = listPos + o, *src = listSrc + o;
            XT acc = b[y];
            int4 p = make_int4(0, 0, 0, 0), r = p;
            if (cnt > 0) {
                p = *(const int4 *)pos;
                r = *(const int4 *)src;
            }
            for (int k = 0; k < cnt; k += 4) {
                int4 pn = p, rn = r;
                if (k + 4 < cnt) {
                    pn = *(const int4 *)(pos + 32 * (k + 4));
                    rn = *(const int4 *)(src + 32 * (k + 4));
                }
                XT v[4], xv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (k + i < cnt) {
                        v[i] = ld<VT, XT>(val, comp(p, i) & 0x7fffffff);
                        xv[i] = x[comp(r, i)];
                    }
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (k + i < cnt) {
                        acc = mac(v[i], xv[i], acc);
                        if (kSymm && comp(p, i) < 0) acc += t;
                    }
                p = pn;
                r = rn;
            }
            b[y] = acc;
        }
    }
    // the launch ends after the long entries' one
    if (numLong && blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Large matrices with short rows: a thread per entry of b on the caller's CRS
// and the plain lists. Nothing of a short list is padding there and twice as
// many threads are resident, which decides where loads in flight do (gatherPlain).
template <typename VT, typename XT, int KER>
__global__ void __launch_bounds__(256)
    kGatherPlain(int n, const int *__restrict__ ptr, const int *__restrict__ entry, const int *__restrict__ src,
                 const int *__restrict__ rowPtr, const int *__restrict__ col, const VT *__restrict__ val,
                 const XT *__restrict__ x, XT *__restrict__ b) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long y = (long long)blockIdx.x * blockDim.x + threadIdx.x; y < n; y += stride) {
        if constexpr (KER == RACE_K_SPMV) {
            XT t = XT(0);
            for (int j = rowPtr[y]; j < rowPtr[y + 1]; ++j) t = mac(ld<VT, XT>(val, j), x[col[j]], t);
            b[y] = t;
        } else {
            XT acc = b[y];
            for (int k = ptr[y]; k < ptr[y + 1]; ++k) {
                const int e = entry[k];
                if (KER == RACE_K_SPMTV || e >= 0) {  // another row's update
                    acc = mac(ld<VT, XT>(val, e), x[src[k]], acc);
                    continue;
                }
                const int s = rowPtr[y], end = rowPtr[y + 1];
                if (end == s) continue;  // a row without entries has no update of its own
                acc = mac(ld<VT, XT>(val, s), x[y], acc);
                XT t = XT(0);
                for (int j = s + 1; j < end; ++j) t = mac(ld<VT, XT>(val, j), x[col[j]], t);
                acc += t;
            }
            b[y] = acc;
        }
    }
}

// Lists of one chunk's entries of b from GatherPlan's, a warp per chunk.
__global__ void kListLayout(int n, int numChunks, const int *__restrict__ len, const int *__restrict__ ptr,
                            const int *__restrict__ entry, const int *__restrict__ src,
                            const int *__restrict__ rowPtr, const long long *__restrict__ off, int *__restrict__ pos,
                            int *__restrict__ srcOut) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const int y = 32 * c + lane;
    if (c >= numChunks || y >= n) return;
    const long long o = off[c] + 4 * lane;
    int k = 0;
    if (len[y] < 0) return;
    for (int i = ptr[y]; i < ptr[y + 1]; ++i) {
        const int e = entry[i];
        if (e < 0 && rowPtr[y] == rowPtr[y + 1]) continue;  // a row without entries has no update of its own
        pos[o + 32 * (k & ~3) + (k & 3)] = e >= 0 ? e : (rowPtr[y] | (int)0x80000000u);
        srcOut[o + 32 * (k & ~3) + (k & 3)] = e >= 0 ? src[i] : y;
        ++k;
    }
}

template <typename VT, typename XT, int KER>
void launchGather(const FuncEntry &f, const DevGather &g, cudaStream_t s) {
    const race_operands &o = f.ops;
    if (o.n == 0) return;
    if (g.plain) {
        kGatherPlain<VT, XT, KER><<<std::min(ceilDiv(o.n, 256), 152 * 16), 256, 0, s>>>(
            o.n, g.ptr, g.entry, g.row, o.rowPtr, o.col, (const VT *)o.val, (const XT *)o.x, (XT *)o.b);
        RACE_CUDA(cudaGetLastError());
        return;
    }
    const GatherArgs a{o.n,     g.numLong,   o.rowPtr,    o.col,       o.val,     o.x,     o.b,       g.len,
                       g.listOff, g.listPos, g.listSrc, g.longY, g.ptr, g.entry, g.row};
    if (a.numLong) {
        kGatherLong<VT, XT, KER><<<ceilDiv(a.numLong, kGatherWarps), kGatherThreads, 0, s>>>(a);
        RACE_CUDA(cudaGetLastError());
    }
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ceilDiv(o.n, kShortThreads));
    cfg.blockDim = dim3(kShortThreads);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = a.numLong ? 1 : 0;  // only behind kGatherLong, whose inputs are complete
    RACE_CUDA(cudaLaunchKernelEx(&cfg, kGather<VT, XT, KER>, o.n, g.numLong, o.rowPtr, o.col, (const VT *)o.val,
                                 (const XT *)o.x, (XT *)o.b, (const int *)g.len, (const long long *)g.listOff,
                                 (const int *)g.listPos, (const int *)g.listSrc));
}

template <typename VT, typename XT>
void launchGatherK(const FuncEntry &f, const DevGather &g, cudaStream_t s) {
    if (f.kernel == RACE_K_SPMV) launchGather<VT, XT, RACE_K_SPMV>(f, g, s);
    else if (f.kernel == RACE_K_SPMTV) launchGather<VT, XT, RACE_K_SPMTV>(f, g, s);
    else launchGather<VT, XT, RACE_K_SYMMSPMV>(f, g, s);
}

}  // namespace

// The number of updates (in an entry's list or its own row) above which a
// warp folds the entry: kLongList, or more where so many entries are longer
// that their folds fill the GPU. A warp's fold issues an instruction per
// update, a thread's shares each with its 31 neighbours, so a matrix whose
// rows are all long wants threads and a few hub rows want warps. Estimated
// cycles of a line, whichever is longest: the folds on the GPU's 608 issue
// queues (an FP64 instruction takes one for 64 cycles; FP32 with its loads
// about 8), the longest fold of a warp (80 and 20 cycles an update) and of a
// thread (140 and 80; measured on lists of up to 28k updates: own rows 100 and
// 52, others' 183 and 105). Measured, 120k rows of 97 entries, with 96 as the
// only line and now: SpMV FP64 608 and 45 us, FP32 65 and 37; SpMTV 618 and 44,
// 131 and 35; 201 entries: 1,245 and 94, 108 and 85 (SpMV); the 50k-row
// power-law graph keeps 96 (SpMV FP64 996 us, by threads alone 1,342; FP32 207
// and 700).
template <typename F>
int foldLine(int n, bool f64, F &&lens) {
    const double issue = (f64 ? 64.0 : 8.0) / 608, warpChain = f64 ? 80 : 20, threadChain = f64 ? 140 : 80;
    struct Line {
        double issue, chain;      // estimated cycles
        long long slots, updates; // of the padded lists and without padding
        int longest;
        double cycles() const { return std::max(issue, chain); }
    };
    auto estimate = [&](int line) {
        long long folds = 0, slots = 0, updates = 0, warpMost = 0, threadMost = 0;
        int longest = 0;
        for (int c = 0; c < n; c += 32) {
            int own = 0, list = 0;
            for (int y = c; y < std::min(n, c + 32); ++y) {
                const auto [o, l] = lens(y);
                longest = std::max(longest, std::max(o, l));
                updates += l;
                if (std::max(o, l) > line) {
                    folds += (long long)o + l;
                    warpMost = std::max(warpMost, (long long)o + l);
                } else {
                    own = std::max(own, o);
                    list = std::max(list, l);
                    threadMost = std::max(threadMost, (long long)o + l);
                }
            }
            folds += own + list;
            slots += 32LL * list;
        }
        return Line{issue * folds, std::max(warpChain * warpMost, threadChain * threadMost), slots, updates, longest};
    };
    int line = kLongList;
    const Line first = estimate(line);
    double best = first.cycles();
    // only the issue queues' time can shrink
    if (first.issue <= first.chain) return line;
    for (int next = line; next < first.longest;) {
        next = next & (next - 1) ? next / 3 * 4 : next / 2 * 3;  // 128, 192, 256, 384, ...
        const Line e = estimate(next);
        if (e.slots > 4 * e.updates) break;  // lists are padded to their chunk's longest
        if (e.cycles() < 0.8 * best) {
            best = e.cycles();
            line = next;
        }
    }
    return line;
}

// Whether kGatherPlain runs a matrix without long entries: from half a million
// rows on (a grid of resident threads then takes more than one turn) and up to
// twelve updates per entry of b. Measured, microseconds with kGather and with
// kGatherPlain, 5-, 7- and 9-point stencils of about 700k rows, and of 1.4 to 2
// million: SpMV FP64 10.6 and 10.3, 14.4 and 12.4, 18.5 and 16.4; 38 and 29, 43
// and 35, 40 and 38; FP32 8.3 and 6.3, 10.4 and 8.3, 10.3 and 10.3; 27 and 17,
// 33 and 24, 27 and 25. SpMTV FP64 25 and 16, 27 and 19, 37 and 30; 62 and 43,
// 59 and 51, 62 and 58; FP32 14.5 and 12.2, 16.5 and 14.5, 23 and 19; 44 and
// 32, 43 and 38, 45 and 40. SymmSpMV FP64 23 and 20, 34 and 31, 41 and 34; 69
// and 50, 77 and 62, 73 and 57; FP32 16.5 and 14.5, 20.0 and 20.6, 20.7 and
// 20.7; 51 and 39, 52 and 45, 47 and 41 (so FP32 with more than six updates
// waits for a million rows). With 360k rows it is the other way round for 9
// points (SymmSpMV FP64 23 and 25, SpMTV FP32 11.8 and 14.2), and for 27-point
// rows at every size (SymmSpMV FP64 753k rows 93 and 144).
bool gatherPlain(int kernel, bool f64, int n, double updates) {
    const bool late = kernel == RACE_K_SYMMSPMV && !f64 && updates > 6;
    return n >= (late ? 1 << 20 : 1 << 19) && updates <= 12;
}

// The device lists of one direction (SpMV: of both) from the host CRS.
void buildGather(Engine &e, FuncEntry &f, int dir, const std::vector<int> &rp, const std::vector<int> &cl) {
    DevGather &g = f.gather[dir];
    const int n = f.ops.n, C = ceilDiv(n, 32);
    const bool lists = f.kernel != RACE_K_SPMV, own = f.kernel != RACE_K_SPMTV;
    const int first = f.kernel == RACE_K_SYMMSPMV ? 1 : 0;
    cudaStream_t s = e.stream;
    GatherOrder go;
    if (lists) go = buildGatherOrder(f.kernel, n, rp.data(), cl.data(), e.phases[dir]);
    const std::vector<int> &ptr = go.ptr;
    auto spread = [&](const std::vector<int> &offsets) {  // shortest and longest
        int lo = INT_MAX, hi = 0;
        const int *p = offsets.data();
        for (int y = 0; y < n; ++y) {
            const int len = p[y + 1] - p[y];
            lo = std::min(lo, len);
            hi = std::max(hi, len);
        }
        return std::pair<int, int>(lo, hi);
    };
    const auto [shortRow, longRow] = own ? spread(rp) : std::pair<int, int>(1, 0);
    const int longList = lists ? spread(ptr).second : 0, most = std::max(longRow - first, longList);
    const long long entries = lists ? ptr[n] : 0;
    const bool f64 = f.ops.vec_type == RACE_VAL_F64;
    const double updates = ((own ? (double)rp[n] - first * (double)n : 0.0) + entries) / std::max(n, 1);
    g.plain = most <= kLongList && gatherPlain(f.kernel, f64, n, updates);
    // Short lists of rows that all have entries are laid out here, straight
    // from the walk; the others on the GPU from the plain ones (kListLayout).
    const bool direct = lists && !g.plain && most <= kLongList && !(first && shortRow == 0);
    std::vector<int> len, longY, pos, src;
    std::vector<long long> listOff;
    long long listSlots = 0;
    GatherPlan gp;
    if (lists && !direct) gp = buildGatherPlan(go, n, rp.data(), cl.data());
    auto lens = [&](int y) {
        return std::pair<int, int>(own ? std::max(0, rp[y + 1] - rp[y] - first) : 0, lists ? ptr[y + 1] - ptr[y] : 0);
    };
    auto cut = [&](int line) {
        for (int c = 0; c < C; ++c) {
            int width = 0;
            for (int y = 32 * c; y < std::min(n, 32 * c + 32); ++y) {
                auto [ownLen, cnt] = lens(y);
                if (std::max(cnt, ownLen) > line) {
                    len[y] = -1;
                    longY.push_back(y);
                    continue;
                }
                if (first && rp[y] == rp[y + 1]) {  // its own update is left out (kListLayout)
                    for (int i = ptr[y]; i < ptr[y + 1]; ++i) cnt -= gp.entry[i] < 0;
                }
                len[y] = cnt;
                width = std::max(width, cnt);
            }
            listOff[c] = listSlots;
            listSlots += 32LL * ((width + 3) & ~3);
        }
    };
    if (direct) {
        len.resize(n);
        listOff.resize(C);
        for (int c = 0; c < C; ++c) {
            const int y0 = 32 * c, y1 = std::min(n, y0 + 32);
            int width = 0;
            for (int y = y0; y < y1; ++y) {
                len[y] = ptr[y + 1] - ptr[y];
                width = std::max(width, len[y]);
            }
            listOff[c] = listSlots;
            listSlots += 32LL * ((width + 3) & ~3);
        }
        pos.resize(listSlots);
        src.resize(listSlots);
        std::vector<long long> next(n);
        for (int y = 0; y < n; ++y) next[y] = listOff[y >> 5] + 4 * (y & 31);
        go.updates(n, rp.data(), cl.data(), [&](int y, int entry, int row) {
            const long long at = next[y];
            pos[at] = entry >= 0 ? entry : (rp[y] | INT_MIN);
            src[at] = row;
            next[y] = at + ((at & 3) == 3 ? 32 * 4 - 3 : 1);  // groups of four per lane
        });
    } else if (!g.plain) {
        len.assign(std::max(n, 1), 0);
        listOff.assign(std::max(C, 1), 0);
        cut(most > kLongList ? foldLine(n, f64, lens) : kLongList);
    }
    // the longest first: a warp each, and the longest bounds the launch
    auto work = [&](int y) {
        return (lists ? ptr[y + 1] - ptr[y] : 0) + (own ? rp[y + 1] - rp[y] : 0);
    };
    std::stable_sort(longY.begin(), longY.end(), [&](int a, int b) { return work(a) > work(b); });
    g.numLong = (int)longY.size();
    // one allocation for all tables (above a megabyte each costs a first call 90 us)
    size_t total = 0;
    auto room = [&](size_t count) {
        const size_t at = total;
        total += (count + 3) & ~(size_t)3;
        return at;
    };
    const size_t plain = gp.entry.size();
    const size_t oOff = room(2 * listOff.size()), oLen = room(len.size()), oLong = room(longY.size()),
                 oPtr = room(gp.ptr.size()), oEntry = room(plain), oRow = room(plain), oPos = room(listSlots),
                 oSrc = room(listSlots);
    g.mem.alloc(total);
    g.listOff = (long long *)(g.mem.p + oOff);
    g.len = g.mem.p + oLen;
    g.longY = g.mem.p + oLong;
    g.ptr = g.mem.p + oPtr;
    g.entry = g.mem.p + oEntry;
    g.row = g.mem.p + oRow;
    g.listPos = g.mem.p + oPos;
    g.listSrc = g.mem.p + oSrc;
    auto put = [&](void *dst, const void *src, size_t bytes) {
        if (bytes) RACE_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
    };
    put(g.len, len.data(), sizeof(int) * len.size());
    put(g.longY, longY.data(), sizeof(int) * longY.size());
    put(g.listOff, listOff.data(), sizeof(long long) * listOff.size());
    if (direct) {
        put(g.listPos, pos.data(), sizeof(int) * pos.size());
        put(g.listSrc, src.data(), sizeof(int) * src.size());
    } else if (lists) {
        put(g.ptr, gp.ptr.data(), sizeof(int) * gp.ptr.size());
        put(g.entry, gp.entry.data(), sizeof(int) * plain);
        put(g.row, gp.row.data(), sizeof(int) * plain);
        if (C > 0 && !g.plain)
            kListLayout<<<ceilDiv(32LL * C, 256), 256, 0, s>>>(n, C, g.len, g.ptr, g.entry, g.row, f.ops.rowPtr, g.listOff,
                                                               g.listPos, g.listSrc);
    }
    RACE_CUDA(cudaGetLastError());
    RACE_CUDA(cudaStreamSynchronize(s));
    g.built = true;
}

// SpMV, SpMTV or SymmSpMV in one launch; the lists of SpMTV and SymmSpMV are
// built at the first call of a direction, SpMV's at its registration.
void runGather(Engine &e, FuncEntry &f, int dir) {
    const race_operands &ops = f.ops;
    if (f.kernel == RACE_K_SPMV) dir = 0;  // its rows are independent
    DevGather &g = f.gather[dir];
    if (!g.built) {
        const int n = ops.n;
        std::vector<int> rp(n + 1);
        RACE_CUDA(cudaMemcpyAsync(rp.data(), ops.rowPtr, sizeof(int) * (n + 1), cudaMemcpyDeviceToHost, e.stream));
        RACE_CUDA(cudaStreamSynchronize(e.stream));
        std::vector<int> cl(std::max(rp[n], 1));
        RACE_CUDA(cudaMemcpyAsync(cl.data(), ops.col, sizeof(int) * (size_t)rp[n], cudaMemcpyDeviceToHost, e.stream));
        RACE_CUDA(cudaStreamSynchronize(e.stream));
        buildGather(e, f, dir, rp, cl);
    }
    if (ops.vec_type == RACE_VAL_F64) {
        if (ops.val_type != RACE_VAL_F64) throw Error(RACE_ERR_INVALID_ARG, "FP64 vectors need FP64 values");
        launchGatherK<double, double>(f, g, e.stream);
    } else if (ops.vec_type == RACE_VAL_F32) {
        if (ops.val_type == RACE_VAL_F32)
            launchGatherK<float, float>(f, g, e.stream);
        else if (ops.val_type == RACE_VAL_BF16)
            launchGatherK<__nv_bfloat16, float>(f, g, e.stream);
        else
            throw Error(RACE_ERR_INVALID_ARG, "FP32 vectors need FP32 or BF16 values");
    } else {
        throw Error(RACE_ERR_INVALID_ARG, "unknown vector type");
    }
}

}  // namespace race
