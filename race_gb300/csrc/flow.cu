// Dataflow execution of the sweeps whose rows depend on one another
// (Gauss-Seidel, Kaczmarz).
//
// RACE's coloring fixes the order of rows that touch the same entries of x
// (src/functionManager.cpp:201-265); everything else may overlap. Instead of
// a grid barrier after every wave or phase of that order, each entry of x
// carries its own state: a copy of x is kept as (value, tag) words that are
// read and written by single 8- or 16-byte accesses, so a reader that sees
// the tag it waits for has the value too, and one row's result reaches a
// dependent row in one L2 store and one L2 load, without fences, flags or
// barriers.
//
// * Gauss-Seidel: tag 1 marks a value of this sweep. A row's entries on rows
//   earlier in the order wait for it (the plan marks those columns with the
//   sign bit); the other entries read a copy of x taken before the sweep, so
//   no row ever waits to overwrite.
// * Kaczmarz: the tag counts the updates made to an entry. A row waits until
//   each of its entries has had exactly the updates of the earlier rows (the
//   plan stores that count per matrix entry) and stores count + 1.
//
// Work is cut into tasks, listed in wave order (waves.cpp), and taken by
// persistent warps from one ticket: a warp holds at most the task it runs
// and the next one, and a task only waits for tasks listed before it, so the
// first unfinished task of the list can always run (the blocks are
// co-resident: cooperative launch). Every wait is bounded.
//
// The arithmetic is that of the wave and leaf executors (sweep.cu), operation
// by operation: which of the two runs is chosen by the same rule, and results
// are the same bit for bit.
//
// What bounds it on GB300 (measured): the chain of dependent rows. One link
// is an L2 store and a load that sees it (850-1100 cycles), the row's FP64
// chain (a warp's FP64 instruction occupies its quarter of the SM for 64
// cycles, whether 1 or 32 lanes are active) and an FP64 division (570
// cycles), about 1.4 us in all. The wave executor took 5.7 us a wave (a grid
// barrier of 152 blocks is 1.25 us, the row data loaded after it the rest),
// the leaf executor one serial row after another in each leaf. Forward +
// backward sweeps, before and after: Gauss-Seidel, 27-point 40x44x41 (leaf
// sums, 248 waves a direction), FP64 2450-2500 and 698-701 us; Kaczmarz, 9-point
// 211x197 (leaf sums, 181 waves) 1150-1170 and 504-508 us; the refinement solve
// of a 100k-row power-law graph (sequential sums, FP32, 24 refinements of two
// sweeps of 315 waves; several graphs) 83-128 and 17-22 ms.
#include <algorithm>
#include <climits>

#include "engine.h"
#include "sweep_ops.cuh"

namespace race {
namespace {

// One block of 8 warps per SM: 1,216 tasks (of up to 4 or 32 rows) in flight,
// several waves of an ordinary matrix, so that a task's row data is loaded
// before its inputs arrive. 4 warps took 2 % more time on the Gauss-Seidel
// pair above, 16 took 16 % more: their polling slows the running rows.
constexpr int kFlowThreads = 256;
constexpr int kFlowWarps = kFlowThreads / 32;

enum FlowKind : int {
    FLOW_CHUNK = 0,  // up to 32 short rows, a thread each: {first position, count, SELL chunk}
    FLOW_ROW = 1,    // one row, a warp folding in order: {position}
    FLOW_LANES = 2,  // leaf arithmetic: {first position, rows, products per lane, 0: one long row}
    FLOW_SEG = 3,    // one segment of a long row: {segment, first entry, end}
    FLOW_SEG0 = 4,   // the same, the row's first segment (its diagonal is left out of a Gauss-Seidel sum)
    FLOW_COMB = 5,   // a long row's segments combined: {position, first segment, end}
    FLOW_SCAT = 6,   // Kaczmarz update of one segment's entries: {row's first segment, first entry, end}
};

// (value, tag) words: 16 bytes for FP64, 8 for FP32, accessed whole.
template <typename XT>
struct TagWord;
template <>
struct TagWord<double> {
    static constexpr int kBytes = 16;
};
template <>
struct TagWord<float> {
    static constexpr int kBytes = 8;
};
__device__ __forceinline__ void ldTag(const void *t, long long i, double &v, int &tag) {
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"((const char *)t + 16 * i)
                 : "memory");
    v = __longlong_as_double((long long)lo);
    tag = (int)hi;
}
__device__ __forceinline__ void stTag(void *t, long long i, double v, int tag) {
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(
                     (char *)t + 16 * i),
                 "l"(__double_as_longlong(v)), "l"((unsigned long long)(unsigned)tag)
                 : "memory");
}
__device__ __forceinline__ void ldTag(const void *t, long long i, float &v, int &tag) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"((const char *)t + 8 * i) : "memory");
    v = __uint_as_float((unsigned)w);
    tag = (int)(w >> 32);
}
__device__ __forceinline__ void stTag(void *t, long long i, float v, int tag) {
    const unsigned long long w = (unsigned long long)__float_as_uint(v) | ((unsigned long long)(unsigned)tag << 32);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"((char *)t + 8 * i), "l"(w) : "memory");
}

struct FlowArgs {
    const int *col;   // the caller's columns
    const void *val;  // the caller's values
    void *x;
    const void *b;
    const int4 *task;
    int numTasks;
    const int4 *pos;  // per plan position: row, first entry, length
    const int *mark;  // per entry: GS: column | earlier row << 31; Kaczmarz: updates to wait for | last update << 31
    void *xt;         // (value, tag) copy of x
    void *xold;       // x before the sweep (Gauss-Seidel)
    void *segDot, *segNrm;  // (value, tag) partial sums per segment; Kaczmarz: segScl the row scale at its first segment
    void *segScl;
    int midRow;       // longer rows are not run by FLOW_CHUNK
    const long long *chunkOff;  // SELL copy of the short rows (sellCol: GS marks), or null
    const void *sellVal;
    const int *sellCol, *sellMark;
    long long maxPolls;  // of one wait
    int *status, *ticket;
};

// The limit of a wait: false once it is passed, or another warp has reported
// one (the status word is then set). The lanes' answers are joined: a lane
// that saw the word before it was set would wait for the others otherwise.
__device__ __forceinline__ bool mayWait(const FlowArgs &a, long long &spins) {
    if ((++spins & 63) != 0) return true;
    int st;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(st) : "l"(a.status) : "memory");
    if (!__any_sync(0xffffffffu, spins > a.maxPolls || st != DEV_OK)) return true;
    atomicCAS(a.status, DEV_OK, DEV_WAIT_TIMEOUT);
    return false;
}

// Waits until the entries of every lane's set bits carry their tags; xv
// receives the values. Called by whole warps, which leave together: after a
// loop that each lane left by itself, every shuffle of the row sums that
// follow took 250 cycles instead of 25 (measured), and with it the chain of
// dependent rows 2.8 us a link instead of 1.8.
template <typename XT, int N>
__device__ __forceinline__ bool await(const FlowArgs &a, const void *words, const int (&idx)[N], const int (&want)[N],
                                      unsigned todo, XT (&xv)[N]) {
    long long spins = 0;
    for (;;) {
        int tag[N];
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (todo >> k & 1) ldTag(words, idx[k], xv[k], tag[k]);
#pragma unroll
        for (int k = 0; k < N; ++k)
            if ((todo >> k & 1) && tag[k] == want[k]) todo &= ~(1u << k);
        if (!__any_sync(0xffffffffu, todo != 0)) return true;
        if (!mayWait(a, spins)) return false;  // the whole warp
    }
}

// The x values of up to N entries of a Gauss-Seidel row (marks m, valid in
// the bits of `valid`): this sweep's value for earlier rows, else the old one.
template <typename XT, int N>
__device__ __forceinline__ bool gsValues(const FlowArgs &a, const int (&m)[N], unsigned valid, XT (&xv)[N]) {
    int c[N], want[N];
    unsigned todo = 0;
#pragma unroll
    for (int k = 0; k < N; ++k) {
        c[k] = m[k] & 0x7fffffff;
        want[k] = 1;
        if (valid >> k & 1) {
            if (m[k] < 0) todo |= 1u << k;
            else xv[k] = ((const XT *)a.xold)[c[k]];
        }
    }
    return await<XT, N>(a, a.xt, c, want, todo, xv);
}

// The x values of up to N entries of a Kaczmarz row (columns c, marks m).
template <typename XT, int N>
__device__ __forceinline__ bool kaczValues(const FlowArgs &a, const int (&c)[N], const int (&m)[N], unsigned valid,
                                           XT (&xv)[N]) {
    int want[N];
#pragma unroll
    for (int k = 0; k < N; ++k) want[k] = m[k] & 0x7fffffff;
    return await<XT, N>(a, a.xt, c, want, valid, xv);
}

// Gauss-Seidel result of row r.
template <typename XT>
__device__ __forceinline__ void gsStore(const FlowArgs &a, int r, XT v) {
    stTag(a.xt, r, v, 1);
    ((XT *)a.x)[r] = v;
}
// A row without entries keeps its value; rows that read it go on.
template <typename XT>
__device__ __forceinline__ void gsKeep(const FlowArgs &a, int r) {
    stTag(a.xt, r, ((const XT *)a.xold)[r], 1);
}
// Kaczmarz update of an entry (mark m of the matrix entry).
template <typename XT>
__device__ __forceinline__ void kaczStore(const FlowArgs &a, int c, int m, XT v) {
    stTag(a.xt, c, v, (m & 0x7fffffff) + 1);
    if (m < 0) ((XT *)a.x)[c] = v;
}

// Up to kBlk entries k0.. of a short row: values, columns and marks, from the
// SELL copy (a lane's entries in groups of four slots) or the caller's CRS.
constexpr int kBlk = 8;
template <typename VT, typename XT, bool KACZ>
__device__ __forceinline__ unsigned shortEntries(const FlowArgs &a, long long off, int lane, int s, int len, int k0,
                                                 XT (&v)[kBlk], int (&c)[kBlk], int (&m)[kBlk]) {
    unsigned valid = 0;
#pragma unroll
    for (int k = 0; k < kBlk; ++k)
        if (k0 + k < len) valid |= 1u << k;
    if (off >= 0) {
#pragma unroll
        for (int g = 0; g < kBlk; g += 4)
            if (k0 + g < len) {
                const long long o = off + 32LL * (k0 + g) + 4 * lane;
                XT vv[4];
                groupVals((const VT *)a.sellVal + o, vv);
                const int4 cc = *(const int4 *)(a.sellCol + o);
                int4 mm = cc;
                if constexpr (KACZ) mm = *(const int4 *)(a.sellMark + o);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    v[g + q] = vv[q];
                    c[g + q] = comp(cc, q);
                    m[g + q] = comp(mm, q);
                }
            }
    } else {
#pragma unroll
        for (int k = 0; k < kBlk; ++k)
            if (valid >> k & 1) {
                v[k] = ld<VT, XT>((const VT *)a.val, s + k0 + k);
                m[k] = a.mark[s + k0 + k];
                c[k] = KACZ ? a.col[s + k0 + k] : m[k];
            }
    }
    return valid;
}

// FLOW_CHUNK: the kernel bodies of kernels.cpp:174-186 (GS) and :285-302
// (KACZ) in their own order, a thread per row. All loops are uniform over the
// warp and lanes meet after every wait: lanes that left a wait at different
// times would otherwise issue the FP64 chain once each, 64 cycles an
// instruction.
template <typename VT, typename XT, bool KACZ>
__device__ __forceinline__ bool chunkTask(const FlowArgs &a, const int4 &t, int lane) {
    const int4 q = lane < t.z ? a.pos[t.y + lane] : make_int4(0, 0, INT_MAX, 0);
    const int r = q.x, s = q.y;
    const bool live = q.z <= a.midRow;
    const int len = live ? q.z : 0;
    const int most = __reduce_max_sync(0xffffffffu, len);
    const long long off = a.chunkOff ? a.chunkOff[t.w] : -1;
    const XT br = live ? ((const XT *)a.b)[r] : XT(1);  // idle lanes divide 1 by 1 (see lanesTask)
    XT v[kBlk], xv[kBlk];
    int c[kBlk], m[kBlk];
    unsigned valid = 0;
    XT sum = KACZ ? -br : br, nrm = XT(0), diag = XT(1);
    for (int k0 = 0; k0 < most; k0 += kBlk) {
        valid = shortEntries<VT, XT, KACZ>(a, off, lane, s, len, k0, v, c, m);
        bool ok;
        if constexpr (KACZ) {
#pragma unroll
            for (int k = 0; k < kBlk; ++k)
                if (valid >> k & 1) nrm = mac(v[k], v[k], nrm);
            ok = kaczValues<XT, kBlk>(a, c, m, valid, xv);
        } else {
            if (k0 == 0) {
                if (len > 0) diag = v[0];
                valid &= ~1u;
            }
            ok = gsValues<XT, kBlk>(a, m, valid, xv);
        }
        if (__any_sync(0xffffffffu, !ok)) return false;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kBlk; ++k)
            if (k0 + k < most)
                if (valid >> k & 1) sum = mac(KACZ ? v[k] : -v[k], xv[k], sum);
    }
    if constexpr (!KACZ) {
        const XT xn = sum / diag;
        if (len > 0) gsStore<XT>(a, r, xn);
        else if (live) gsKeep<XT>(a, r);
    } else {
        const XT sc = sum / (len > 0 ? nrm : XT(1));
        for (int k0 = 0; k0 < most; k0 += kBlk) {
            if (most > kBlk) {  // the block's entries again (only this row may change their x values)
                valid = shortEntries<VT, XT, true>(a, off, lane, s, len, k0, v, c, m);
                kaczValues<XT, kBlk>(a, c, m, valid, xv);
                __syncwarp();
            }
#pragma unroll
            for (int k = 0; k < kBlk; ++k)
                if (valid >> k & 1) kaczStore<XT>(a, c[k], m[k], mac(-sc, v[k], xv[k]));
        }
    }
    return true;
}

// Entries of a row staged per warp for an in-order fold: every lane gathers
// its share, then all lanes read the (value, x) pairs as broadcasts.
template <typename XT>
constexpr int kFoldPer = sizeof(XT) == 8 ? 4 : 8;  // entries per lane and round (32 KB of shared memory a block)

template <typename XT>
struct FlowStage {
    XT v[kFlowWarps][32 * kFoldPer<XT>];
    XT x[kFlowWarps][32 * kFoldPer<XT>];
};

// FLOW_ROW: the same bodies, the row's entries gathered by a warp and folded
// in order (every lane runs the whole chain).
template <typename VT, typename XT, bool KACZ>
__device__ __forceinline__ bool rowTask(const FlowArgs &a, FlowStage<XT> &st, const int4 &t, int lane) {
    constexpr int P = kFoldPer<XT>;
    const int4 q = a.pos[t.y];
    const int r = q.x, s = q.y, e = q.y + q.z, w = threadIdx.x >> 5;
    const VT *val = (const VT *)a.val;
    const XT br = ((const XT *)a.b)[r];
    XT sum = KACZ ? -br : br, nrm = XT(0);
    for (int jr = KACZ ? s : s + 1; jr < e; jr += 32 * P) {
        XT v[P], xv[P];
        int c[P], m[P];
        unsigned valid = 0;
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const int j = jr + 32 * k + lane;
            v[k] = xv[k] = XT(0);
            c[k] = m[k] = 0;
            if (j < e) {
                valid |= 1u << k;
                v[k] = ld<VT, XT>(val, j);
                m[k] = a.mark[j];
                if constexpr (KACZ) c[k] = a.col[j];
            }
        }
        bool ok;
        if constexpr (KACZ) ok = kaczValues<XT, P>(a, c, m, valid, xv);
        else ok = gsValues<XT, P>(a, m, valid, xv);
        if (__any_sync(0xffffffffu, !ok)) return false;
        __syncwarp();  // the previous round's reads are done
#pragma unroll
        for (int k = 0; k < P; ++k) {
            st.v[w][32 * k + lane] = v[k];
            st.x[w][32 * k + lane] = xv[k];
        }
        __syncwarp();
        const int cnt = min(32 * P, e - jr);
#pragma unroll 8
        for (int i = 0; i < cnt; ++i) {
            if constexpr (KACZ) {
                sum = mac(st.v[w][i], st.x[w][i], sum);
                nrm = mac(st.v[w][i], st.v[w][i], nrm);
            } else {
                sum = mac(-st.v[w][i], st.x[w][i], sum);
            }
        }
    }
    if constexpr (!KACZ) {
        if (lane == 0) {
            if (e == s) gsKeep<XT>(a, r);
            else gsStore<XT>(a, r, sum / ld<VT, XT>(val, s));
        }
    } else {
        const XT sc = sum / nrm;
        for (int j = s + lane; j < e; j += 32) {
            const int c = a.col[j], m = a.mark[j];
            XT xv;
            int tag;
            ldTag(a.xt, c, xv, tag);  // read above with the awaited tag, and only this row may change it
            kaczStore<XT>(a, c, m, mac(-sc, ld<VT, XT>(val, j), xv));
        }
    }
    __syncwarp();
    return true;
}

// The leaf executor's sum of up to 32 products, one per lane and an xor
// butterfly over 16, 8, 4, 2, 1, by 8 lanes holding E products each (lane l
// those of lanes l, l+8, ...): the first two steps are additions within a
// lane. Absent products are zeros.
template <typename XT, int E>
__device__ __forceinline__ XT lanesSum(const XT (&p)[E]) {
    XT t;
    if constexpr (E == 4) t = (p[0] + p[2]) + (p[1] + p[3]);
    else if constexpr (E == 2) t = p[0] + p[1];
    else t = p[0];
#pragma unroll
    for (int o = 4; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

// FLOW_LANES, rows of up to 8 E products: the leaf executor's row, 8 lanes
// each, four rows per warp, so that an FP64 instruction serves four rows.
template <typename VT, typename XT, bool KACZ, int E>
__device__ __forceinline__ bool lanesTask(const FlowArgs &a, const int4 &t, int lane) {
    const int sub = lane >> 3, l = lane & 7;
    const bool live = sub < t.z;
    const int4 q = live ? a.pos[t.y + sub] : make_int4(0, 0, 0, 0);
    const int r = q.x, s = q.y, e = q.y + q.z;
    const VT *val = (const VT *)a.val;
    // Idle lanes divide 1 by 1: a zero numerator sends the whole warp through
    // the FP64 division's special cases (775 us instead of 692 us for the
    // Gauss-Seidel pair above, 559 instead of 511 us for the Kaczmarz pair).
    const XT br = live ? ((const XT *)a.b)[r] : XT(1);
    XT diag = XT(1), v[E], xv[E], p[E];
    if constexpr (!KACZ)
        if (e > s) diag = ld<VT, XT>(val, s);
    int c[E], m[E];
    unsigned valid = 0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
        const int j = s + (KACZ ? 0 : 1) + 8 * k + l;
        v[k] = xv[k] = XT(0);
        c[k] = m[k] = 0;
        if (j < e) {
            valid |= 1u << k;
            v[k] = ld<VT, XT>(val, j);
            m[k] = a.mark[j];
            if constexpr (KACZ) c[k] = a.col[j];
        }
    }
    XT nrm = XT(1);
    bool ok;
    if constexpr (KACZ) {
#pragma unroll
        for (int k = 0; k < E; ++k) p[k] = mac(v[k], v[k], XT(0));
        nrm = lanesSum<XT, E>(p);
        ok = kaczValues<XT, E>(a, c, m, valid, xv);
    } else {
        ok = gsValues<XT, E>(a, m, valid, xv);
    }
    if (__any_sync(0xffffffffu, !ok)) return false;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < E; ++k) p[k] = mac(KACZ ? v[k] : -v[k], xv[k], XT(0));
    const XT dot = lanesSum<XT, E>(p);
    if constexpr (!KACZ) {
        const XT xn = (br + dot) / diag;
        if (live && l == 0) {
            if (e > s) gsStore<XT>(a, r, xn);
            else gsKeep<XT>(a, r);
        }
    } else {
        const XT sc = (dot - br) / (e > s ? nrm : XT(1));
#pragma unroll
        for (int k = 0; k < E; ++k) {
            const XT xn = mac(-sc, v[k], xv[k]);
            if (valid >> k & 1) kaczStore<XT>(a, c[k], m[k], xn);
        }
    }
    return true;
}

// FLOW_LANES, one longer row: lanes stride it, then the butterfly.
template <typename VT, typename XT, bool KACZ>
__device__ __forceinline__ bool lanesRow(const FlowArgs &a, const int4 &t, int lane) {
    const int4 q = a.pos[t.y];
    const int r = q.x, s = q.y, e = q.y + q.z;
    const VT *val = (const VT *)a.val;
    constexpr int U = 4;
    const XT br = ((const XT *)a.b)[r];
    XT dot = XT(0), nrm = XT(0), v[U], xv[U];
    int c[U], m[U];
    for (int j0 = KACZ ? s : s + 1; j0 < e; j0 += 32 * U) {
        unsigned valid = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + 32 * u + lane;
            if (j < e) {
                valid |= 1u << u;
                v[u] = ld<VT, XT>(val, j);
                m[u] = a.mark[j];
                if constexpr (KACZ) c[u] = a.col[j];
            }
        }
        bool ok;
        if constexpr (KACZ) ok = kaczValues<XT, U>(a, c, m, valid, xv);
        else ok = gsValues<XT, U>(a, m, valid, xv);
        if (__any_sync(0xffffffffu, !ok)) return false;
        __syncwarp();
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (valid >> u & 1) {
                dot = mac(KACZ ? v[u] : -v[u], xv[u], dot);
                if constexpr (KACZ) nrm = mac(v[u], v[u], nrm);
            }
    }
    dot = warpSum(dot);
    if constexpr (!KACZ) {
        const XT xn = (br + dot) / ld<VT, XT>(val, s);
        if (lane == 0) gsStore<XT>(a, r, xn);
    } else {
        const XT sc = (dot - br) / warpSum(nrm);
        for (int j = s + lane; j < e; j += 32) {
            const int cj = a.col[j], mj = a.mark[j];
            XT xj;
            int tag;
            ldTag(a.xt, cj, xj, tag);  // read above with the awaited tag, and only this row may change it
            kaczStore<XT>(a, cj, mj, mac(-sc, ld<VT, XT>(val, j), xj));
        }
    }
    return true;
}

// FLOW_SEG / FLOW_SEG0: partial sums of a long row's segment.
template <typename VT, typename XT, bool KACZ>
__device__ __forceinline__ bool segTask(const FlowArgs &a, const int4 &t, int lane, bool first) {
    constexpr int P = kHugeSeg / 32;
    const VT *val = (const VT *)a.val;
    XT v[P], xv[P];
    int c[P], m[P];
    unsigned valid = 0;
#pragma unroll
    for (int k = 0; k < P; ++k) {
        const int j = t.z + lane + 32 * k;
        v[k] = xv[k] = XT(0);
        c[k] = m[k] = 0;
        if (j < t.w && !(!KACZ && first && j == t.z)) {
            valid |= 1u << k;
            v[k] = ld<VT, XT>(val, j);
            m[k] = a.mark[j];
            if constexpr (KACZ) c[k] = a.col[j];
        }
    }
    bool ok;
    if constexpr (KACZ) ok = kaczValues<XT, P>(a, c, m, valid, xv);
    else ok = gsValues<XT, P>(a, m, valid, xv);
    if (__any_sync(0xffffffffu, !ok)) return false;
    XT dot = XT(0), nrm = XT(0);
#pragma unroll
    for (int k = 0; k < P; ++k) {
        dot = mac(v[k], xv[k], dot);
        if constexpr (KACZ) nrm = mac(v[k], v[k], nrm);
    }
    dot = warpSum(dot);
    if constexpr (KACZ) nrm = warpSum(nrm);
    if (lane == 0) {
        if constexpr (KACZ) stTag(a.segNrm, t.y, nrm, 1);
        stTag(a.segDot, t.y, dot, 1);
    }
    return true;
}

// FLOW_COMB: the segments of a long row in a fixed order, then its update.
template <typename VT, typename XT, bool KACZ>
__device__ __forceinline__ bool combTask(const FlowArgs &a, const int4 &t, int lane) {
    const int4 q = a.pos[t.y];
    const XT br = ((const XT *)a.b)[q.x];
    const XT diag = ld<VT, XT>((const VT *)a.val, q.y);
    XT S = XT(0), Q = XT(0);
    for (int g0 = t.z; g0 < t.w; g0 += 32) {
        const int idx[1] = {g0 + lane}, want[1] = {1};
        const unsigned todo = g0 + lane < t.w;
        XT p[1] = {XT(0)}, q2[1] = {XT(0)};
        bool ok = await<XT, 1>(a, a.segDot, idx, want, todo, p);
        if constexpr (KACZ) ok = await<XT, 1>(a, a.segNrm, idx, want, todo, q2) && ok;
        if (__any_sync(0xffffffffu, !ok)) return false;
        __syncwarp();
        S += p[0];
        if constexpr (KACZ) Q += q2[0];
    }
    S = warpSum(S);
    if constexpr (KACZ) Q = warpSum(Q);
    if (lane == 0) {
        if constexpr (KACZ) stTag(a.segScl, t.z, (S - br) / Q, 1);
        else gsStore<XT>(a, q.x, (br - S) / diag);
    }
    return true;
}

// FLOW_SCAT: Kaczmarz update of a segment's entries with the row's scale. The
// segment's sum read the same words with their tags, but in another warp, and
// relaxed accesses to the scale's word carry no order for these: the entries
// are awaited again.
template <typename VT, typename XT>
__device__ __forceinline__ bool scatTask(const FlowArgs &a, const int4 &t, int lane) {
    const int idx[1] = {t.y}, want[1] = {1};
    XT sc[1];
    const bool ok = await<XT, 1>(a, a.segScl, idx, want, 1u, sc);
    if (__any_sync(0xffffffffu, !ok)) return false;
    constexpr int P = 4;
    for (int j0 = t.z; j0 < t.w; j0 += 32 * P) {
        XT v[P], xv[P];
        int c[P], m[P];
        unsigned valid = 0;
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const int j = j0 + 32 * k + lane;
            v[k] = xv[k] = XT(0);
            c[k] = m[k] = 0;
            if (j < t.w) {
                valid |= 1u << k;
                v[k] = ld<VT, XT>((const VT *)a.val, j);
                c[k] = a.col[j];
                m[k] = a.mark[j];
            }
        }
        if (__any_sync(0xffffffffu, !kaczValues<XT, P>(a, c, m, valid, xv))) return false;
#pragma unroll
        for (int k = 0; k < P; ++k)
            if (valid >> k & 1) kaczStore<XT>(a, c[k], m[k], mac(-sc[0], v[k], xv[k]));
    }
    return true;
}

template <typename VT, typename XT, bool KACZ>
__global__ void __launch_bounds__(kFlowThreads, 1) kFlow(FlowArgs a) {
    __shared__ FlowStage<XT> stage;
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * kFlowWarps;
    // behind a sweep that gave up and has not been reported yet nothing runs
    // (read along with the first task: no round trip of its own)
    int st;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(st) : "l"(a.status) : "memory");
    int it = (blockIdx.x * kFlowThreads + threadIdx.x) >> 5;
    while (it < a.numTasks) {
        int next = 0;
        if (lane == 0) next = nw + atomicAdd(a.ticket, 1);  // the round trip overlaps this task
        const int4 t = a.task[it];
        if (__any_sync(0xffffffffu, st != DEV_OK)) return;
        bool ok = true;
        switch (t.x) {
        case FLOW_CHUNK: ok = chunkTask<VT, XT, KACZ>(a, t, lane); break;
        case FLOW_ROW: ok = rowTask<VT, XT, KACZ>(a, stage, t, lane); break;
        case FLOW_LANES:
            ok = t.w == 1   ? lanesTask<VT, XT, KACZ, 1>(a, t, lane)
                 : t.w == 2 ? lanesTask<VT, XT, KACZ, 2>(a, t, lane)
                 : t.w == 4 ? lanesTask<VT, XT, KACZ, 4>(a, t, lane)
                            : lanesRow<VT, XT, KACZ>(a, t, lane);
            break;
        case FLOW_SEG:
        case FLOW_SEG0: ok = segTask<VT, XT, KACZ>(a, t, lane, t.x == FLOW_SEG0); break;
        case FLOW_COMB: ok = combTask<VT, XT, KACZ>(a, t, lane); break;
        default:
            if constexpr (KACZ) ok = scatTask<VT, XT>(a, t, lane);
            break;
        }
        if (!ok) return;
        it = __shfl_sync(0xffffffffu, next, 0);
    }
}

// Start of a sweep: the (value, tag) copy of x with tags 0, the old x of a
// Gauss-Seidel sweep, the segments' tags and the ticket.
template <typename XT, bool KACZ>
__global__ void __launch_bounds__(256) kFlowPrep(int n, int numSegs, const XT *__restrict__ x, void *xt,
                                                 XT *__restrict__ xold, void *segDot, void *segNrm, void *segScl,
                                                 int *ticket) {
    const long long i0 = blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 == 0) *ticket = 0;
    for (long long i = i0; i < n; i += gridDim.x * blockDim.x) {
        const XT v = x[i];
        if constexpr (!KACZ) xold[i] = v;
        stTag(xt, i, v, 0);
    }
    for (long long i = i0; i < numSegs; i += gridDim.x * blockDim.x) {
        stTag(segDot, i, XT(0), 0);
        if constexpr (KACZ) {
            stTag(segNrm, i, XT(0), 0);
            stTag(segScl, i, XT(0), 0);
        }
    }
}

// GS marks: a column whose row comes earlier in the order gets the sign bit.
__global__ void kGsMarks(int n, const int *__restrict__ rowPtr, const int *__restrict__ col,
                         const int *__restrict__ order, int *__restrict__ mark) {
    const long long r = warpOf(blockIdx.x, blockDim.x, threadIdx.x);
    if (r >= n) return;
    const int o = order[r];
    for (int j = rowPtr[r] + (threadIdx.x & 31); j < rowPtr[r + 1]; j += 32) {
        const int c = col[j];
        mark[j] = order[c] < o ? (c | (int)0x80000000u) : c;
    }
}

template <typename VT, typename XT, bool KACZ>
void launchFlow(Engine &e, FuncEntry &f, int dir, bool leaf) {
    static const int resident = [] {
        int dev = 0, sms = 0, occ = 0;
        RACE_CUDA(cudaGetDevice(&dev));
        RACE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        RACE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kFlow<VT, XT, KACZ>, kFlowThreads, 0));
        return occ > 0 ? sms : 1;
    }();
    const race_operands &o = f.ops;
    DevFlow &w = f.flow[dir];
    const DevWaves &wv = f.waves[dir];
    const int n = o.n, S = wv.numSegs, T = w.numTasks[leaf];
    constexpr size_t word = TagWord<XT>::kBytes;
    char *seg = (char *)w.segWords.p;
    int *ticket = f.flowTicket.p;
    if (T == 0) return;
    const int prepBlocks = std::min(ceilDiv(std::max(n, S), 256), 152 * 8);
    kFlowPrep<XT, KACZ><<<prepBlocks, 256, 0, e.stream>>>(n, S, (const XT *)o.x, f.flowX.p, (XT *)f.flowOld.p, seg,
                                                          seg + word * S, seg + 2 * word * S, ticket);
    RACE_CUDA(cudaGetLastError());
    FlowArgs a{o.col, o.val, o.x, o.b, w.task[leaf].p, T, w.pos.p, w.mark.p, f.flowX.p, f.flowOld.p,
               seg, seg + word * S, seg + 2 * word * S, wv.sellMidRow,
               wv.sell ? wv.chunkOff.p : nullptr, wv.sellVal.p, wv.sellCol.p, w.sellMark.p, e.sweepMaxPolls, e.dStatus.p, ticket};
    void *args[] = {&a};
    const int blocks = std::max(1, std::min(resident, ceilDiv(T, kFlowWarps)));
    RACE_CUDA(cudaLaunchCooperativeKernel((void *)kFlow<VT, XT, KACZ>, blocks, kFlowThreads, args, 0, e.stream));
}

template <typename VT, typename XT>
void launchFlowK(Engine &e, FuncEntry &f, int dir, bool leaf) {
    if (f.kernel == RACE_K_GS) launchFlow<VT, XT, false>(e, f, dir, leaf);
    else launchFlow<VT, XT, true>(e, f, dir, leaf);
}

}  // namespace

// The task lists of one direction: `ptr`, `rows`, `huge` and the segments are
// the wave plan's (rows sorted by length inside ordinary waves), chunkOf the
// SELL chunk of every 32nd position of an ordinary wave.
void buildFlow(Engine &e, FuncEntry &f, int dir, const FlowOrder &fo, const std::vector<int> &rp,
               const std::vector<int> &ptr, const std::vector<int> &rows, const std::vector<unsigned char> &huge,
               const std::vector<int> &segFirst, const std::vector<int> &segBeg, const std::vector<int> &segEnd,
               const std::vector<int> &waveChunk) {
    DevFlow &w = f.flow[dir];
    w.ok = fo.ok;
    if (!fo.ok) return;
    const int n = f.ops.n, mid = f.waves[dir].sellMidRow;
    const bool kacz = f.kernel == RACE_K_KACZ;
    auto len = [&](int p) { return rp[rows[p] + 1] - rp[rows[p]]; };
    std::vector<int4> pos(rows.size());
    for (size_t p = 0; p < rows.size(); ++p) pos[p] = make_int4(rows[p], rp[rows[p]], len((int)p), 0);
    std::vector<int4> seq, leaf;
    for (size_t wi = 0; wi < huge.size(); ++wi) {
        const int p0 = ptr[wi], p1 = ptr[wi + 1];
        if (huge[wi]) {
            for (int p = p0; p < p1; ++p)
                for (int g = segFirst[p]; g < segFirst[p + 1]; ++g)
                    seq.push_back(make_int4(g == segFirst[p] ? FLOW_SEG0 : FLOW_SEG, g, segBeg[g], segEnd[g]));
            for (int p = p0; p < p1; ++p) seq.push_back(make_int4(FLOW_COMB, p, segFirst[p], segFirst[p + 1]));
            if (kacz)
                for (int p = p0; p < p1; ++p)
                    for (int g = segFirst[p]; g < segFirst[p + 1]; ++g)
                        seq.push_back(make_int4(FLOW_SCAT, segFirst[p], segBeg[g], segEnd[g]));
        } else {
            for (int p = p0; p < p1; ++p)
                if (len(p) > mid) seq.push_back(make_int4(FLOW_ROW, p, 0, 0));
            for (int p = p0; p < p1; p += 32) {
                const int cnt = std::min(32, p1 - p);
                bool any = false;
                for (int q = p; q < p + cnt; ++q) any |= len(q) <= mid;
                if (any) seq.push_back(make_int4(FLOW_CHUNK, p, cnt, waveChunk.at(wi) + (p - p0) / 32));
            }
        }
        // leaf arithmetic: four neighbouring rows of up to 32 products per
        // warp, longer rows alone
        auto perLane = [&](int q) {
            const int terms = len(q) - (kacz ? 0 : 1);
            return terms <= 8 ? 1 : terms <= 16 ? 2 : terms <= 32 ? 4 : 0;
        };
        for (int p = p0; p < p1;) {
            const int k = perLane(p);
            int cnt = 1, most = k;
            while (k && cnt < 4 && p + cnt < p1 && perLane(p + cnt)) most = std::max(most, perLane(p + cnt++));
            leaf.push_back(make_int4(FLOW_LANES, p, cnt, most));
            p += cnt;
        }
    }
    cudaStream_t s = e.stream;
    w.numTasks[0] = (int)seq.size();
    w.numTasks[1] = (int)leaf.size();
    w.task[0].upload(seq.empty() ? nullptr : seq.data(), std::max<size_t>(seq.size(), 1), s);
    w.task[1].upload(leaf.empty() ? nullptr : leaf.data(), std::max<size_t>(leaf.size(), 1), s);
    w.pos.upload(pos.empty() ? nullptr : pos.data(), std::max<size_t>(pos.size(), 1), s);
    const size_t word = f.ops.vec_type == RACE_VAL_F64 ? 16 : 8;
    w.segWords.alloc(std::max<size_t>(3 * word * segBeg.size(), 16));
    f.flowX.ensure(std::max<size_t>(word * n, 16));
    if (!kacz) f.flowOld.ensure(std::max<size_t>(word / 2 * n, 16));
    f.flowTicket.ensure(1);
    const size_t nnz = std::max(rp[n], 1);
    if (kacz) {
        w.mark.upload(fo.mark.empty() ? nullptr : fo.mark.data(), nnz, s);
        RACE_CUDA(cudaStreamSynchronize(s));
    } else {
        w.mark.alloc(nnz);
        DevBuf<int> order;
        order.upload(fo.order.empty() ? nullptr : fo.order.data(), std::max(n, 1), s);
        if (n > 0) kGsMarks<<<ceilDiv(32LL * n, 256), 256, 0, s>>>(n, f.ops.rowPtr, f.ops.col, order.p, w.mark.p);
        RACE_CUDA(cudaGetLastError());
        RACE_CUDA(cudaStreamSynchronize(s));
    }
}

// One direction of a Gauss-Seidel or Kaczmarz function; leaf: the leaf
// executor's sums, else the sequential ones.
void runFlow(Engine &e, FuncEntry &f, int dir, bool leaf) {
    const race_operands &o = f.ops;
    if (o.vec_type == RACE_VAL_F64) {
        if (o.val_type != RACE_VAL_F64) throw Error(RACE_ERR_INVALID_ARG, "FP64 vectors need FP64 values");
        launchFlowK<double, double>(e, f, dir, leaf);
    } else if (o.vec_type == RACE_VAL_F32) {
        if (o.val_type == RACE_VAL_F32) launchFlowK<float, float>(e, f, dir, leaf);
        else if (o.val_type == RACE_VAL_BF16) launchFlowK<__nv_bfloat16, float>(e, f, dir, leaf);
        else throw Error(RACE_ERR_INVALID_ARG, "FP32 vectors need FP32 or BF16 values");
    } else {
        throw Error(RACE_ERR_INVALID_ARG, "unknown vector type");
    }
}

}  // namespace race
