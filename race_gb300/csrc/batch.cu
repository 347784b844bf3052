// Block matrix-power kernel over many right-hand sides and many matrices in
// one persistent launch.
//
// A block-MPK function is RACE's matrix power (src/matrixPower.cpp level
// groups, executor src/functionManager.cpp:618-823) applied to nrhs vectors
// at once: x_k[r][j] = sum_c A[r][c] x_{k-1}[c][j] for j < nrhs, with x
// stored power-major, then row, then right-hand side (one 8- or 4-byte
// element per right-hand side, consecutive), so a row's nrhs values are one
// contiguous segment. The reference has no multi-vector or multi-matrix
// form: each RACE::Interface runs one matrix with one vector.
//
// Thread mapping: R = nrhs lanes per row (R in {1,2,4,8,16,32}), 32/R rows
// per warp pass. Each lane walks its row's CRS entries in order as a
// sequential fused multiply-add chain, so every right-hand side is computed
// exactly like a single-vector SpMV (MAT_SPMV_KERNEL's order,
// examples/src/helpers/kernels.cpp:749-777): FP64 results are bit-identical
// to p sequential fma SpMVs per right-hand side. The lanes of one row read
// the same value and column (a broadcast) and R consecutive x entries.
//
// Schedule: chunks of a few dozen rows inside level groups (blockChunkRows);
// a work item is (power, chunk). The chunks of all members are numbered
// through, and the items are listed by c + k lag (k the power, c the chunk):
// power k of a chunk follows its power k-1 by `lag` chunks, as many as the
// GPU has in flight and more than any chunk's inputs lie ahead of it, so that
// inputs are complete when an item is taken, and the list holds every item
// after its inputs. Persistent warps take items from a global ticket; an item
// waits (bounded) for the chunks of the previous power its columns fall in.
// Dependencies stay inside a member and point to earlier tickets, so the
// launch cannot deadlock. A batch is one memset of the completion flags plus
// one kernel, and can be captured once in a CUDA graph and replayed.
//
// Measured on GB300, p = 4 (before: items of 32 rows, one member's powers
// right behind one another, so that most warps waited): 24 matrices of 100^2
// to 500^2, 8 FP32 right-hand sides, 587 and 254 us; 16 of 100^2 to 700^2, 16
// FP64 ones, 2,015 and 1,832 us, 94 % of the FP64 pipe's time (1.08 G fma at 2
// a cycle and SM); one of about 120^2, 16 FP32 ones, 47 and 39 us.
#include <algorithm>

#include <cuda_bf16.h>

#include "engine.h"

namespace race {

bool chunkDependencyRanges(const int *rowPtr, const int *col, const std::vector<int> &chunkRow,
                           const std::vector<int> &chunkGroup, std::vector<int> &range, cudaStream_t s);

namespace {

constexpr int kBlockThreads = 256;

__device__ __forceinline__ int ldAcquireB(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ldRelaxedB(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Rows that a warp takes at once, and the most rows of an item: 4 KB of one
// power's right-hand sides, 32 to 128 rows. Each item costs a ticket (one
// address for the whole GPU), its table entry, the poll of its inputs and a
// release; 32 rows of 8 FP32 right-hand sides are less work than that.
int blockPassRows(int nrhs, int vecType) {
    return 32 / std::max(1, nrhs * (vecType == RACE_VAL_F64 ? 8 : 4) / 16);
}
int blockMaxRows(int nrhs, int vecType) {
    const int rows = 4096 / (nrhs * (vecType == RACE_VAL_F64 ? 8 : 4));
    return std::min(128, std::max(32, rows & ~31));
}
// Whether a batch's items mostly wait for one another (kMpkBlock, FEW): up to
// three chunks for four warps, and with long rows, whose chain of loads is the
// item's time, up to four chunks a warp. Measured, the other form / FEW, p = 8
// unless noted: 7-point 40^3, one FP64 right-hand side (2,000 chunks) 120 and
// 101 us; 9-point 300^2, 8 FP32 ones (5,600) 108 and 101; 27-point 50^3, one FP64
// (3,900) 385 and 298, 16 FP32 (15,600) 319 and 292; 5- and 9-point 250^2, 16
// FP32, p = 4 (8,100) 41 and 43; 16 of 100^2 to 500^2, 8 BF16, p = 4, 8 % more.
bool latencyBound(int chunks, int warps, double entriesPerRow) {
    return 4LL * chunks <= 3LL * warps || (entriesPerRow > 16 && chunks <= 4LL * warps);
}
// Rows of an item where `rows` rows in all are shared by `warps` warps: whole
// passes, so that every warp has some before any takes more than one pass.
// Measured with the most rows throughout instead: 5 matrices of 100^2 to
// 200^2 with 8 FP64 right-hand sides 154 us (115 us with 32 rows).
int blockItemRows(long long rows, int warps, int nrhs, int vecType) {
    const int pass = blockPassRows(nrhs, vecType);
    const long long share = rows / std::max(warps, 1) / pass * pass;
    return (int)std::min<long long>(blockMaxRows(nrhs, vecType), std::max<long long>(pass, share));
}

__device__ __forceinline__ double mulAdd(double v, double x, double acc) { return fma(v, x, acc); }
__device__ __forceinline__ float mulAdd(float v, float x, float acc) { return fmaf(v, x, acc); }
__device__ __forceinline__ float mulAdd(__nv_bfloat16 v, float x, float acc) {
    return fmaf(__bfloat162float(v), x, acc);
}

struct BlockArgs {
    const BlockMember *members;
    // three per item: {first row, end row, member, power}, then three chunk
    // ranges [lo, hi] read at the previous power and the item's own chunk:
    // {lo0, hi0, lo1, hi1}, {lo2, hi2, chunk, 0}
    const int4 *item;
    int numItems, numChunks;
    int *done, *ticket, *status;
};

// V consecutive right-hand sides of one row as one 16-byte (or smaller)
// vector access.
template <typename XT, int V>
struct alignas(sizeof(XT) * V) XVec {
    XT v[V];
};

// Right-hand sides per lane: one 16-byte access (FP64: 2, FP32: 4), at most R.
template <typename XT, int R>
__host__ __device__ constexpr int kVecOf() {
    return R < (int)(16 / sizeof(XT)) ? R : (int)(16 / sizeof(XT));
}

// Rows [r0, r1) (at most 32) of one member at power k -> k+1, all right-hand
// sides. A lane owns V consecutive right-hand sides of one row (R/V lanes per
// row, 32V/R rows per pass) and runs one sequential fma chain per right-hand
// side over the row's entries in CRS order. The rows' offsets are read once
// per range by one coalesced load and passed around by shuffles. U entries'
// loads are in flight at a time: two where the L1 decides (four keep 13 % fewer
// warps' x rows there: 254 and 281 us for the FP32 batch above), four where the
// latency of a row does (kMpkBlock, FEW).
template <typename VT, typename XT, int R, int U>
__device__ __forceinline__ void blockRows(const BlockMember &m, int r0, int r1, int k) {
    constexpr int V = kVecOf<XT, R>();
    constexpr int L = R / V;        // lanes per row
    constexpr int RPP = 32 / L;     // rows per pass
    using Vec = XVec<XT, V>;
    const int lane = threadIdx.x & 31;
    const int sub = lane / L, q = lane % L;
    const int nr = r1 - r0;
    const VT *__restrict__ val = (const VT *)m.val;
    const int *__restrict__ col = m.col;
    const XT *xin = (const XT *)m.x + (size_t)k * m.n * R + q * V;
    XT *xout = (XT *)m.x + (size_t)(k + 1) * m.n * R + q * V;
    const int rs = lane < nr ? m.rowPtr[r0 + lane] : 0;
    const int rEnd = m.rowPtr[r1];
    for (int base = 0; base < nr; base += RPP) {
        const int i = base + sub;
        const int e0 = __shfl_sync(0xffffffffu, rs, min(i, 31));
        const int eNext = __shfl_sync(0xffffffffu, rs, min(i + 1, 31));
        if (i < nr) {
            const int e1 = i + 1 < nr ? eNext : rEnd;
            Vec acc;
#pragma unroll
            for (int t = 0; t < V; ++t) acc.v[t] = XT(0);
#pragma unroll U
            for (int e = e0; e < e1; ++e) {
                const VT a = val[e];
                const Vec xv = *reinterpret_cast<const Vec *>(xin + (size_t)col[e] * R);
#pragma unroll
                for (int t = 0; t < V; ++t) acc.v[t] = mulAdd(a, xv.v[t], acc.v[t]);
            }
            *reinterpret_cast<Vec *>(xout + (size_t)(r0 + i) * R) = acc;
        }
    }
}

// Relaxed polls, one acquire fence after the successful one (an acquire load
// per flag empties the L1 each time) and a warp barrier behind the fence. FEW
// (few chunks, so that most items wait for their inputs and one latency follows
// another): acquire loads, which unlike the fence do not wait for the warp's
// own stores.
template <typename VT, typename XT, int R, bool FEW>
__global__ void __launch_bounds__(kBlockThreads) kMpkBlock(BlockArgs a) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(a.ticket, 1);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= a.numItems) return;
        const int4 h = a.item[3 * (size_t)it], d0 = a.item[3 * (size_t)it + 1], d1 = a.item[3 * (size_t)it + 2];
        const int k = h.w;
        const BlockMember m = a.members[h.z];
        if (k > 0) {
            const int *done = a.done + (size_t)(k - 1) * a.numChunks;
            auto set = [&](int i) { return (FEW ? ldAcquireB(done + i) : ldRelaxedB(done + i)) != 0; };
            long long spins = 0;
            for (;;) {
                bool ok = true;
                for (int i = d0.x + lane; i <= d0.y; i += 32) ok &= set(i);
                for (int i = d0.z + lane; i <= d0.w; i += 32) ok &= set(i);
                for (int i = d1.x + lane; i <= d1.y; i += 32) ok &= set(i);
                if (__all_sync(0xffffffffu, ok)) break;
                if (++spins > kSpinLimit || ldAcquireB(a.status) != DEV_OK) {
                    if (lane == 0) atomicCAS(a.status, DEV_OK, DEV_WAIT_TIMEOUT);
                    return;
                }
                __nanosleep(32);
            }
            if (!FEW) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            __syncwarp();  // a lane reads what other lanes' flags stand for; the vote orders nothing
        }
        for (int r = h.x; r < h.y; r += 32) blockRows<VT, XT, R, FEW ? 4 : 2>(m, r, min(h.y, r + 32), k);
        __syncwarp();
        if (lane == 0)
            asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(a.done + (size_t)k * a.numChunks + d1.z), "r"(1)
                         : "memory");
    }
}

// Plain x_{k+1} = A x_k for all right-hand sides of one member (the
// p-launch baseline on the same data).
template <typename VT, typename XT, int R>
__global__ void __launch_bounds__(kBlockThreads) kSpmvBlock(BlockMember m, int k) {
    const int warps = gridDim.x * (blockDim.x >> 5);
    const int rowsPerWarp = 32;
    for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); (long long)w * rowsPerWarp < m.n; w += warps)
        blockRows<VT, XT, R, 4>(m, w * rowsPerWarp, min(m.n, (w + 1) * rowsPerWarp), k);
}

template <typename K>
int residentBlocksOf(K kernel) {
    int dev = 0, sms = 0, occ = 0;
    RACE_CUDA(cudaGetDevice(&dev));
    RACE_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    RACE_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kBlockThreads, 0));
    return sms * std::max(occ, 1);
}

template <typename VT, typename XT, int R, bool FEW = false>
int blockResident() {
    static const int blocks = residentBlocksOf(kMpkBlock<VT, XT, R, FEW>);
    return blocks;
}
template <typename VT, typename XT, int R>
void launchBlock(const BlockArgs &a, bool few, cudaStream_t s) {
    if (few) kMpkBlock<VT, XT, R, true><<<blockResident<VT, XT, R, true>(), kBlockThreads, 0, s>>>(a);
    else kMpkBlock<VT, XT, R, false><<<blockResident<VT, XT, R>(), kBlockThreads, 0, s>>>(a);
}

template <typename VT, typename XT, int R>
void launchSpmv(const BlockMember &m, int k, cudaStream_t s) {
    static const int blocks = residentBlocksOf(kSpmvBlock<VT, XT, R>);
    const int need = ceilDiv(ceilDiv(m.n, 32), kBlockThreads / 32);
    kSpmvBlock<VT, XT, R><<<std::max(1, std::min(blocks, need)), kBlockThreads, 0, s>>>(m, k);
}

// Type and width dispatch: (FP64 values, FP64 x), (FP32, FP32), (BF16, FP32).
template <template <typename, typename, int> class Fn, typename... A>
void dispatch(int valType, int vecType, int nrhs, A &&...args) {
    auto byWidth = [&](auto tag) {
        using VT = typename decltype(tag)::first_type;
        using XT = typename decltype(tag)::second_type;
        switch (nrhs) {
        case 1: Fn<VT, XT, 1>::run(args...); break;
        case 2: Fn<VT, XT, 2>::run(args...); break;
        case 4: Fn<VT, XT, 4>::run(args...); break;
        case 8: Fn<VT, XT, 8>::run(args...); break;
        case 16: Fn<VT, XT, 16>::run(args...); break;
        case 32: Fn<VT, XT, 32>::run(args...); break;
        default: throw Error(RACE_ERR_INVALID_ARG, "nrhs must be 1, 2, 4, 8, 16 or 32");
        }
    };
    if (valType == RACE_VAL_F64 && vecType == RACE_VAL_F64) byWidth(std::pair<double, double>{});
    else if (valType == RACE_VAL_F32 && vecType == RACE_VAL_F32) byWidth(std::pair<float, float>{});
    else if (valType == RACE_VAL_BF16 && vecType == RACE_VAL_F32) byWidth(std::pair<__nv_bfloat16, float>{});
    else throw Error(RACE_ERR_INVALID_ARG, "block MPK types: FP64 values with FP64 x, or FP32/BF16 values with FP32 x");
}

template <typename VT, typename XT, int R>
struct LaunchBlockFn {
    static void run(const BlockArgs &a, bool few, cudaStream_t s) { launchBlock<VT, XT, R>(a, few, s); }
};
template <typename VT, typename XT, int R>
struct WarpsInFlightFn {
    static void run(int &warps) { warps = blockResident<VT, XT, R>() * (kBlockThreads / 32); }
};
template <typename VT, typename XT, int R>
struct LaunchSpmvFn {
    static void run(const BlockMember &m, int k, cudaStream_t s) { launchSpmv<VT, XT, R>(m, k, s); }
};

// Warps of a batch launch: its items in flight.
int blockWarpsInFlight(int valType, int vecType, int nrhs) {
    int warps = 0;
    dispatch<WarpsInFlightFn>(valType, vecType, nrhs, warps);
    return warps;
}

}  // namespace

void validateBlockTypes(int valType, int vecType, int nrhs) {
    if (!((valType == RACE_VAL_F64 && vecType == RACE_VAL_F64) ||
          ((valType == RACE_VAL_F32 || valType == RACE_VAL_BF16) && vecType == RACE_VAL_F32)))
        throw Error(RACE_ERR_INVALID_ARG, "block MPK types: FP64 values with FP64 x, or FP32/BF16 values with FP32 x");
    if (nrhs != 1 && nrhs != 2 && nrhs != 4 && nrhs != 8 && nrhs != 16 && nrhs != 32)
        throw Error(RACE_ERR_INVALID_ARG, "nrhs must be 1, 2, 4, 8, 16 or 32");
}

void buildBatchTables(BatchTables &t, const std::vector<const BlockPlan *> &plans, cudaStream_t s) {
    if (plans.empty()) throw Error(RACE_ERR_INVALID_ARG, "empty batch");
    const BlockPlan &p0 = *plans[0];
    t.valType = p0.valType;
    t.vecType = p0.vecType;
    t.nrhs = p0.nrhs;
    t.maxPower = 0;
    std::vector<BlockMember> mem;
    long long rows = 0, entries = 0;
    for (const BlockPlan *p : plans) {
        if (p->valType != t.valType || p->vecType != t.vecType || p->nrhs != t.nrhs)
            throw Error(RACE_ERR_INCOMPATIBILITY, "batch members differ in value type, vector type or nrhs");
        t.maxPower = std::max(t.maxPower, p->power);
        mem.push_back(BlockMember{p->ops.rowPtr, p->ops.col, p->ops.val, p->ops.x, p->n, p->power});
        rows += p->n;
        entries += p->entries;
    }
    // A batch's chunks: consecutive chunks of a member's plan and level group
    // put together up to the rows that the whole batch leaves each warp.
    const int warps = blockWarpsInFlight(t.valType, t.vecType, t.nrhs);
    const int limit = blockItemRows(rows, warps, t.nrhs, t.vecType);
    struct Chunk {
        int row0, row1, member;
        int lo[3], hi[3];  // chunks read (empty: [0, -1])
    };
    std::vector<Chunk> chunks;
    int reach = 0;
    for (size_t m = 0; m < plans.size(); ++m) {
        const BlockPlan &p = *plans[m];
        const size_t before = chunks.size();
        std::vector<int> of(p.numChunks);  // chunk of the batch
        for (int c = 0; c < p.numChunks; ++c) {
            const bool join = chunks.size() > before && c > 0 && p.chunkGroup[c] == p.chunkGroup[c - 1] &&
                              p.chunkRow[c + 1] - chunks.back().row0 <= limit;
            if (join) chunks.back().row1 = p.chunkRow[c + 1];
            else chunks.push_back(Chunk{p.chunkRow[c], p.chunkRow[c + 1], (int)m, {0, 0, 0}, {-1, -1, -1}});
            of[c] = (int)chunks.size() - 1;
        }
        for (int c = 0; c < p.numChunks; ++c)
            for (int d = 0; d < 3; ++d) {
                const int lo = p.depRange[6 * (size_t)c + 2 * d], hi = p.depRange[6 * (size_t)c + 2 * d + 1];
                if (hi < lo) continue;
                Chunk &u = chunks[of[c]];
                u.lo[d] = u.hi[d] < 0 ? of[lo] : std::min(u.lo[d], of[lo]);
                u.hi[d] = std::max(u.hi[d], of[hi]);
                reach = std::max(reach, of[hi] - of[c]);
            }
    }
    const int base = (int)chunks.size();
    t.numMembers = (int)plans.size();
    t.numChunks = base;
    // items by c + k lag (a lag of all chunks already is power by power);
    // twice the warps in flight: 281 us instead of 287 us at once that many
    const int lag = std::max(1, std::min(base, std::max(reach + 1, 2 * warps)));
    t.few = latencyBound(base, warps, entries / (double)std::max<long long>(rows, 1));
    std::vector<int4> item;
    size_t total = 0;
    for (const Chunk &u : chunks) total += plans[u.member]->power;
    item.reserve(3 * std::max<size_t>(total, 1));
    for (long long at = 0; at < base + (long long)(t.maxPower - 1) * lag; ++at)
        for (int k = (int)std::min<long long>(at / lag, t.maxPower - 1); k >= 0; --k) {
            const long long c = at - (long long)k * lag;
            if (c >= base) break;
            const Chunk &u = chunks[c];
            if (k >= plans[u.member]->power) continue;
            item.push_back(make_int4(u.row0, u.row1, u.member, k));
            item.push_back(make_int4(u.lo[0], u.hi[0], u.lo[1], u.hi[1]));
            item.push_back(make_int4(u.lo[2], u.hi[2], (int)c, 0));
        }
    t.numItems = (int)(item.size() / 3);
    t.members.upload(mem.data(), mem.size(), s);
    t.item.upload(item.empty() ? nullptr : item.data(), std::max<size_t>(item.size(), 1), s);
    t.done.alloc(std::max<size_t>((size_t)t.maxPower * t.numChunks, 1));
    t.ticket.alloc(1);
    t.status.alloc(1);
    RACE_CUDA(cudaMemsetAsync(t.status.p, 0, sizeof(int), s));
    RACE_CUDA(cudaStreamSynchronize(s));
}

std::unique_ptr<BlockPlan> buildBlockPlan(Engine &e, const race_operands &ops, int power, int nrhs) {
    validateBlockTypes(ops.val_type, ops.vec_type, nrhs);
    // lanes read up to 16 bytes of consecutive right-hand sides at once
    const size_t xs = ops.vec_type == RACE_VAL_F64 ? 8 : 4;
    const size_t vecBytes = std::min<size_t>(16, xs * nrhs);
    if (reinterpret_cast<uintptr_t>(ops.x) % vecBytes != 0)
        throw Error(RACE_ERR_INVALID_ARG, "block MPK x must be aligned to min(16, nrhs * element size) bytes");
    auto plan = std::make_unique<BlockPlan>();
    plan->n = ops.n;
    plan->nrhs = nrhs;
    plan->power = power;
    plan->valType = ops.val_type;
    plan->vecType = ops.vec_type;
    plan->ops = ops;
    const std::vector<int> &gp = e.groupPtr;
    const int G = (int)gp.size() - 1;
    std::vector<int> chunkGroup;
    plan->chunkRow.assign(1, 0);
    const int rows =
        blockItemRows(ops.n, blockWarpsInFlight(ops.val_type, ops.vec_type, nrhs), nrhs, ops.vec_type);
    for (int g = 0; g < G; ++g)
        for (int r = gp[g]; r < gp[g + 1]; r += rows) {
            plan->chunkRow.push_back(std::min(gp[g + 1], r + rows));
            chunkGroup.push_back(g);
        }
    const int C = (int)chunkGroup.size();
    plan->numChunks = C;
    plan->chunkGroup = chunkGroup;
    plan->entries = e.nnz;
    if (!chunkDependencyRanges(ops.rowPtr, ops.col, plan->chunkRow, chunkGroup, plan->depRange, e.stream))
        throw Error(RACE_ERR_INVALID_ARG,
                    "MPK operand is not in the engine's level order (permute it with getPerm/getInvPerm)");
    buildBatchTables(plan->tables, {plan.get()}, e.stream);
    return plan;
}

// Resets the completion flags, ticket and status word and launches the
// persistent kernel: all stream-ordered, so the sequence can be captured.
void runBatch(BatchTables &t, int *status, cudaStream_t s) {
    RACE_CUDA(cudaMemsetAsync(t.done.p, 0, sizeof(int) * (size_t)t.maxPower * t.numChunks, s));
    RACE_CUDA(cudaMemsetAsync(t.ticket.p, 0, sizeof(int), s));
    if (t.numItems == 0) return;
    BlockArgs a{t.members.p, t.item.p, t.numItems, t.numChunks, t.done.p, t.ticket.p, status};
    dispatch<LaunchBlockFn>(t.valType, t.vecType, t.nrhs, a, t.few, s);
    RACE_CUDA(cudaGetLastError());
}

void runBlockSpmv(const BlockPlan &p, int k, cudaStream_t s) {
    const BlockMember m{p.ops.rowPtr, p.ops.col, p.ops.val, p.ops.x, p.n, p.power};
    if (p.n == 0) return;
    dispatch<LaunchSpmvFn>(p.valType, p.vecType, p.nrhs, m, k, s);
    RACE_CUDA(cudaGetLastError());
}

}  // namespace race
