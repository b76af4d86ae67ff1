// Expert-parallel dispatch on one rank: every row's final place is this rank's own output.
//
// The general kernel (ep_kernels.cu) shares its launch with peers: counts travel as epoch-tagged units, rows through the window
// of their destination, a receive step takes them out, and the pointers of every route's destination live in registers next to
// it.  Without peers none of that is needed, and what remains is
//
//   1. route the block's tokens (or take the given ids), rank the routes within the block, write the block's counts;
//   2. one barrier among the blocks;
//   3. every block reads the counts of all blocks, a column (expert) at a time: sixteen blocks' one-byte counts per lane and load,
//      so that all columns are on their way at once.  The sum over all blocks, scanned over the columns, says where a column's
//      rows start; the sum over the blocks before this one says where this block's rows start in it;
//   4. a warp per token (or per part of one, in small batches) converts the row once and stores it to all its places.
//
// A batch of a few tokens takes a handful of blocks in one cluster: the counts are read out of the blocks' shared memory behind a
// cluster barrier, and the launch needs no cooperative form, no table, and no counters that have to be cleared (16 x 7168 by 256 experts, fp8
// 16.2 us with the barrier in memory, 10.0 so; 64 tokens 17.8 and 14.8; 40 x 4096, top-6, 16 bits 11.5 and 8.9).
//
// Bound by the stores of step 4 for large batches; steps 1 to 3 are a chain of memory round trips that small batches wait for
// (us, general kernel and this one: 16 x 7168 by 256 experts, fp8 18.3 14.6; 1009 x 4096, top-6, 16 bits 23.5 17.2; 4096 x 7168, fp8 91 80, of
// which the stores take 63: 3.9 TB/s of writes, what a plain fill of such a buffer reaches.  The reads of the tokens pass beside them; brought to
// L2 during steps 1 to 3 they only delay the routes, 89).
// The blocks wait for one another, so the launch is a cooperative one.
#include <cuda_runtime_api.h>

#include "device/tilexr_convert.cuh"
#include "device/tilexr_perf_trace.cuh"
#include "device/tilexr_rma.cuh"
#include "device/tilexr_sync.cuh"
#include "ep_device.cuh"
#include "ep_kernels.cuh"
#include "tilexr_ep.h"

namespace TileXR {

using namespace tilexr;

namespace {

struct LocalSmem {
    int32_t *routeExpert;   // [routesPerBlock]  expert or -1
    int32_t *routeRank;     // [routesPerBlock]  rank among the block's routes to the same expert
    float *routeWeight;     // [routesPerBlock]
    int32_t *hist;          // [E] routes of this block per expert
    int32_t *before;        // [E] routes of earlier blocks per expert; later first row of this block's routes to it
    int32_t *colPrefix;     // [E + 1] routes of all blocks to the experts before e
    int32_t *groupSum;      // [32]
};

__device__ __forceinline__ LocalSmem CarveLocalSmem(uint8_t *base, int E, int routesPerBlock)
{
    LocalSmem s;
    s.routeExpert = reinterpret_cast<int32_t *>(base);
    s.routeRank = s.routeExpert + routesPerBlock;
    s.routeWeight = reinterpret_cast<float *>(s.routeRank + routesPerBlock);
    s.hist = reinterpret_cast<int32_t *>(s.routeWeight + routesPerBlock);
    s.before = s.hist + E;
    s.colPrefix = s.before + E;
    s.groupSum = s.colPrefix + E + 1;
    return s;
}

// 32 bytes to a 32-byte boundary (whole sectors; two 16-byte stores per lane would each touch every sector of the row's piece).
__device__ __forceinline__ void StoreVec32(uint8_t *p, const Vec16 &lo, const Vec16 &hi)
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y),
                 "r"(hi.z), "r"(hi.w)
                 : "memory");
}

// Sum of the first `n` (0 to 16 / sizeof(COUNT)) counts of a 16-byte vector.
template <typename COUNT>
__device__ __forceinline__ uint32_t SumCounts(const uint4 &v, int n)
{
    const uint32_t words[4] = {v.x, v.y, v.z, v.w};
    uint32_t sum = 0;
    constexpr int PER_WORD = 4 / sizeof(COUNT);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int have = max(0, min(PER_WORD, n - i * PER_WORD));
        const uint32_t mask = have == PER_WORD ? 0xffffffffu : (1u << (have * 8 * static_cast<int>(sizeof(COUNT)))) - 1u;
        const uint32_t w = words[i] & mask;
        if (sizeof(COUNT) == 1) sum = __dp4a(w, 0x01010101u, sum);
        else sum += (w & 0xffffu) + (w >> 16);
    }
    return sum;
}

// Totals of all blocks (into sm.colPrefix[e + 1]) and of the blocks before this one (sm.before[e]) for every column.
template <typename COUNT>
__device__ __forceinline__ void SumColumns(const uint8_t *table, int pitch, int E, int G, int block, const LocalSmem &sm, int warp, int lane)
{
    constexpr int PER_VEC = 16 / sizeof(COUNT);
    constexpr int AT_ONCE = 4;
    const int vecs = (G + PER_VEC - 1) / PER_VEC;
    for (int e0 = warp; e0 < E; e0 += EP_WARPS * AT_ONCE) {
        uint32_t all[AT_ONCE] = {0u, 0u, 0u, 0u}, mine[AT_ONCE] = {0u, 0u, 0u, 0u};
        for (int v0 = 0; v0 < vecs; v0 += 32) {
            const int v = v0 + lane;
            uint4 q[AT_ONCE];
#pragma unroll
            for (int i = 0; i < AT_ONCE; ++i) {
                const int e = e0 + i * EP_WARPS;
                q[i] = make_uint4(0u, 0u, 0u, 0u);
                if (v < vecs && e < E) q[i] = __ldcg(reinterpret_cast<const uint4 *>(table + static_cast<int64_t>(e) * pitch) + v);
            }
            const int first = v * PER_VEC;
#pragma unroll
            for (int i = 0; i < AT_ONCE; ++i) {
                all[i] += SumCounts<COUNT>(q[i], G - first);
                mine[i] += SumCounts<COUNT>(q[i], block - first);
            }
        }
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) {
            const int e = e0 + i * EP_WARPS;
            all[i] = __reduce_add_sync(0xffffffffu, all[i]);
            mine[i] = __reduce_add_sync(0xffffffffu, mine[i]);
            if (lane == 0 && e < E) {
                sm.colPrefix[e + 1] = static_cast<int32_t>(all[i]);
                sm.before[e] = static_cast<int32_t>(mine[i]);
            }
        }
    }
}

// `block`'s counts into column-major rows of `pitch` bytes.
template <typename COUNT>
__device__ __forceinline__ void StoreCounts(uint8_t *table, int pitch, int E, int block, const int32_t *hist, int tid)
{
    for (int e = tid; e < E; e += EP_BLOCK_THREADS) {
        reinterpret_cast<COUNT *>(table + static_cast<int64_t>(e) * pitch)[block] = static_cast<COUNT>(hist[e]);
    }
}

// The same out of the shared memory of the cluster's blocks.
__device__ __forceinline__ void SumColumnsOfCluster(int E, int G, int block, const LocalSmem &sm, int tid)
{
    for (int e = tid; e < E; e += EP_BLOCK_THREADS) {
        const uint32_t mineAddr = SmemAddr(sm.hist + e);
        int all = 0, mine = 0;
#pragma unroll 8
        for (int b = 0; b < G; ++b) {
            uint32_t remote;
            int v;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mineAddr), "r"(b));
            asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
            all += v;
            if (b < block) mine += v;
        }
        sm.colPrefix[e + 1] = all;
        sm.before[e] = mine;
    }
}

template <int TRANSPORT, bool CLUSTER>
__device__ void DispatchLocalBody(const EpDispatchArgs &a)
{
    if (CLUSTER) {
        StreamRelease();
        StreamWait();
    }
    extern __shared__ __align__(16) uint8_t smemRaw[];
    CommArgs *comm = a.comm;
    Waiter w = MakeWaiter(comm, a.magic, blockIdx.x);
    const int E = a.numExperts;
    const int K = a.topK;
    const int G = gridDim.x;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int block = blockIdx.x;
    LocalSmem sm = CarveLocalSmem(smemRaw, E, static_cast<int>(a.tokensPerBlock) * K);
    PerfScope perf = PerfInit(tid == 0 ? a.perfTrace : nullptr, static_cast<uint32_t>(comm->rank), block);
    PerfStageBegin(perf, TILEXR_PERF_KERNEL_TOTAL);
    PerfStageBegin(perf, TILEXR_PERF_CHUNK_TOTAL);
    // counts [E][pitch] in the rank's own window; launches of one communicator follow one another, so one half serves all of them
    const bool wide = static_cast<int>(a.tokensPerBlock) * K > 255;
    const int pitch = (G * (wide ? 2 : 1) + 15) & ~15;
    uint8_t *table = DataHalf(comm, comm->rank, 0) + a.win.blockCountOff;
    // [0] blocks that have counted, over all launches; [1] how many that were before this one.  Block 0 moves [1] on once everybody has arrived, so
    // nothing is cleared at the end and no block has to be the last to leave (1009 x 4096, top-6, 16 bits 21.0 -> 18.4 us; 4096 x 7168, fp8 83.6 -> 80.9).
    uint32_t *doneBlocks = reinterpret_cast<uint32_t *>(CtrlWord(comm, comm->rank, TILEXR_CTRL_SCRATCH_WORD + EP_SCRATCH_LOCAL_DONE_WORD));
    const uint32_t doneBefore = !CLUSTER && tid == 0 ? __ldcg(doneBlocks + 1) : 0u;

    if (block == 0 && tid == 0) {
        comm->dfx[TILEXR_DFX_MAGIC] = w.epoch;
        comm->dfx[TILEXR_DFX_OP] = TILEXR_OP_EP_DISPATCH;
        comm->dfx[TILEXR_DFX_COUNT_ARG] = a.bs;
        comm->dfx[TILEXR_DFX_RUN_STATUS] = TILEXR_RUN_STARTED;
        if (a.laneCountOut != nullptr) *a.laneCountOut = 0;
    }
    const int t0 = min(a.bs, static_cast<int>(block * a.tokensPerBlock));
    const int nTok = min(a.bs, t0 + static_cast<int>(a.tokensPerBlock)) - t0;
    const int nRoutes = nTok * K;
    const uint64_t inBytes = static_cast<uint64_t>(a.h) * a.elemSize;      // of a token
    const uint64_t rowBytes = a.win.rowBytes;                              // of a row of the output

    // ---- 1. route, rank, count ---------------------------------------------------------------------------------
    for (int e = tid; e < E; e += EP_BLOCK_THREADS) sm.hist[e] = 0;
    for (int i = warp; i < nTok; i += EP_WARPS) {
        const int t = t0 + i;
        const int64_t route = static_cast<int64_t>(t) * K + lane;
        int e = -1;
        float weight = 1.0f;
        if (a.gateLogits != nullptr) {
            e = RouteToken(a.gateLogits + static_cast<int64_t>(t) * E, a.selectionBias, E, K, a.scoreFunc, a.renormalize, a.routedScale, lane,
                           a.topkIdsOut + static_cast<int64_t>(t) * K, a.topkWeightsOut + static_cast<int64_t>(t) * K, &weight);
        } else if (lane < K) {
            e = a.expertIds[route];
            if (a.expertScales != nullptr) weight = a.expertScales[route];
        }
        if (lane < K) {
            if (e < 0 || e >= E) e = -1;
            if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_TOKEN && a.activeMask[t] == 0) e = -1;
            if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_EXPERT && a.activeMask[route] == 0) e = -1;
            sm.routeExpert[i * K + lane] = e;
            sm.routeWeight[i * K + lane] = weight;
            if (a.gateLogits == nullptr && a.topkIdsOut != nullptr) a.topkIdsOut[route] = e;
        }
    }
    __syncthreads();
    if (warp == 0) RankBlockRoutes(nRoutes, sm.routeExpert, sm.routeRank, sm.hist, lane);
    __syncthreads();
    if (!CLUSTER) {
        if (wide) StoreCounts<uint16_t>(table, pitch, E, block, sm.hist, tid);
        else StoreCounts<uint8_t>(table, pitch, E, block, sm.hist, tid);
        __syncthreads();
    }
    PerfStageEnd(perf, TILEXR_PERF_CHUNK_TOTAL);
    PerfStageBegin(perf, TILEXR_PERF_POST_SYNC);

    // ---- 2. all blocks have counted ----------------------------------------------------------------------------
    PerfStageBegin(perf, TILEXR_PERF_CHUNK_BARRIER);
    bool ok = true;
    if (CLUSTER) {
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        bool got = true;
        if (tid == 0) {
            __threadfence();
            atom_add_acq_rel_gpu_u32(doneBlocks, 1u);
            uint32_t polls = 0;
            while (ld_acquire_gpu_u32(doneBlocks) - doneBefore < static_cast<uint32_t>(G)) {
                if ((++polls & 63u) == 0) {
                    const uint64_t t = now_ns();
                    if (w.deadline == 0) {
                        w.deadline = t + comm->waitTimeoutNs;
                    } else if (t > w.deadline || AbortRaised(w)) {
                        RaiseFailure(w, TILEXR_DEV_GRID_BARRIER_TIMEOUT, comm->rank, block, static_cast<uint64_t>(G), ld_acquire_gpu_u32(doneBlocks) - doneBefore);
                        got = false;
                        break;
                    }
                }
            }
        }
        ok = BlockBroadcastOk(got);
    }
    PerfStageEnd(perf, TILEXR_PERF_CHUNK_BARRIER);

    // ---- 3. where the rows go ----------------------------------------------------------------------------------
    if (ok) {
        if (CLUSTER) SumColumnsOfCluster(E, G, block, sm, tid);
        else if (wide) SumColumns<uint16_t>(table, pitch, E, G, block, sm, warp, lane);
        else SumColumns<uint8_t>(table, pitch, E, G, block, sm, warp, lane);
        __syncthreads();
        if (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // this block has read the others' counts
        // prefix sums of the totals: warps scan 32 columns each, then every warp scans the (at most 32) sums of those
        const int groups32 = (E + 31) / 32;
        for (int c = warp; c < groups32; c += EP_WARPS) {
            int v = c * 32 + lane < E ? sm.colPrefix[c * 32 + lane + 1] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            if (c * 32 + lane < E) sm.colPrefix[c * 32 + lane + 1] = v;
            if (lane == 31) sm.groupSum[c] = v;
        }
        if (tid == 0) sm.colPrefix[0] = 0;
        __syncthreads();
        {
            const int own = lane < groups32 ? sm.groupSum[lane] : 0;
            int v = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            for (int c = warp; c < groups32; c += EP_WARPS) {
                const int groupBefore = __shfl_sync(0xffffffffu, v - own, c);
                if (c * 32 + lane < E) sm.colPrefix[c * 32 + lane + 1] += groupBefore;
            }
        }
        __syncthreads();
        for (int e = tid; e < E; e += EP_BLOCK_THREADS) sm.before[e] += sm.colPrefix[e];
        bool fits = true;
        if (tid == 0) {
            fits = sm.colPrefix[E] <= static_cast<int64_t>(a.maxRecvRows);
            if (!fits) RaiseFailure(w, TILEXR_DEV_BAD_ARGUMENT, 0, 0, a.maxRecvRows, static_cast<uint64_t>(sm.colPrefix[E]));
        }
        ok = BlockBroadcastOk(fits);
    }
    PerfStageEnd(perf, TILEXR_PERF_POST_SYNC);

    // ---- 4. the rows -------------------------------------------------------------------------------------------
    PerfStageBegin(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC);
    if (ok) {
        const bool bf16 = a.isBf16 != 0;
        constexpr bool mx = TRANSPORT == EP_MXFP8;
        constexpr bool round = TRANSPORT == EP_FP8_ROUND;
        constexpr bool quant = mx || round || TRANSPORT == EP_FP8;
        const bool mxE5m2 = a.quantMode == TileXREp::TILEXR_EP_QUANT_MXFP8_E5M2;
        const bool int8Dynamic = a.quantMode == TileXREp::TILEXR_EP_QUANT_DYNAMIC_INT8;
        const int chunks = a.h / 16;             // 16 elements per lane and iteration (8-bit transports)
        const int iters = (chunks + 31) / 32;
        uint8_t *scalesOut = reinterpret_cast<uint8_t *>(a.dynamicScalesOut);
        // A block with few tokens (small batches) cuts every token into column ranges for several warps.
        const int parts = nTok > 0 ? max(1, min(iters, static_cast<int>(EP_WARPS) / nTok)) : 1;
        for (int item = warp; item < nTok * parts; item += EP_WARPS) {
            const int i = item / parts;
            const int part = item % parts;
            const int t = t0 + i;
            const uint8_t *row = a.x + static_cast<int64_t>(t) * inBytes;
            // lane k owns route k of this token
            int myExpert = -1;
            uint32_t myRow = 0;
            if (lane < K) {
                myExpert = sm.routeExpert[i * K + lane];
                if (myExpert >= 0) myRow = static_cast<uint32_t>(sm.before[myExpert] + sm.routeRank[i * K + lane]);
                if (a.routeRowsOut != nullptr && part == 0) a.routeRowsOut[static_cast<int64_t>(t) * K + lane] = myExpert >= 0 ? static_cast<int32_t>(myRow) : -1;
            }
            const uint32_t routes = __ballot_sync(0xffffffffu, myExpert >= 0);
            if (routes == 0) continue;
            if (TRANSPORT == EP_INT8) {
                // every route is quantised for its own expert: one pass for the row's amax (dynamic), one to convert
                for (uint32_t m = routes; m != 0; m &= m - 1) {
                    const int k = __ffs(m) - 1;
                    const uint32_t rr = __shfl_sync(0xffffffffu, myRow, k);
                    const int e = __shfl_sync(0xffffffffu, myExpert, k);
                    uint8_t *p = a.expandXOut + rr * rowBytes;
                    const float *sc = a.quantScales != nullptr ? a.quantScales + static_cast<int64_t>(e) * a.h : nullptr;
                    float inv = 1.0f;
                    if (int8Dynamic) {
                        const float amax = Int8RowAmax(row, sc, chunks, bf16, lane);
                        if (amax > 0.f) inv = 127.0f / amax;
                        if (part == 0 && lane == 0) a.dynamicScalesOut[rr] = amax > 0.f ? amax / 127.0f : 1.0f;
                    }
                    Int8RowStore(row, sc, inv, chunks, bf16, part, parts, lane, p);
                }
            } else if (quant) {
                // each 512-element chunk is quantised once and stored to every destination right away
#pragma unroll 2
                for (int it = part; it < iters; it += parts) {
                    const int c = it * 32 + lane;
                    float f[16];
                    if (c < chunks) {
                        Unpack8(ld_vec16(row + static_cast<int64_t>(c) * 32), bf16, f);
                        Unpack8(ld_vec16(row + static_cast<int64_t>(c) * 32 + 16), bf16, f + 8);
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j) f[j] = 0.f;
                    }
                    Vec16 sv;
                    if (round) {
                        // what the receiver of the 8-bit row would make of it, 32 bytes per lane
                        float own;
                        const Vec16 q = QuantFp8Block16(f, &sv, &own);
                        Fp8Unpack8(make_uint2(q.x, q.y), __NV_E4M3, own, f);
                        Fp8Unpack8(make_uint2(q.z, q.w), __NV_E4M3, own, f + 8);
                        const Vec16 lo = Pack8(f, bf16), hi = Pack8(f + 8, bf16);
                        uint8_t *dst = a.expandXOut + static_cast<int64_t>(c) * 32;
                        for (uint32_t m = routes; m != 0; m &= m - 1) {
                            const uint32_t rr = __shfl_sync(0xffffffffu, myRow, __ffs(m) - 1);
                            if (c < chunks) StoreVec32(dst + rr * rowBytes, lo, hi);
                        }
                        continue;
                    }
                    const Vec16 q = mx ? QuantMx16(f, mxE5m2, lane, &sv) : QuantFp8Block16(f, &sv);
                    // this iteration's 16 bytes of the scale row: lane k stores them for route k
                    if ((routes >> lane) & 1u) st_vec16(scalesOut + static_cast<uint64_t>(myRow) * a.win.scaleRowBytes + it * 16, sv);
                    uint8_t *dst = a.expandXOut + static_cast<int64_t>(c) * 16;
                    for (uint32_t m = routes; m != 0; m &= m - 1) {
                        const uint32_t rr = __shfl_sync(0xffffffffu, myRow, __ffs(m) - 1);
                        if (c < chunks) st_vec16(dst + rr * rowBytes, q);
                    }
                }
            } else {
                const uint64_t perPart = ((rowBytes + parts - 1) / parts + 511) & ~511ull;
                const uint64_t b0 = min(rowBytes, perPart * part);
                const uint64_t nBytes = min(rowBytes - b0, perPart);
                if ((reinterpret_cast<uintptr_t>(row) & 15u) == 0) {       // the output and its rows are on the 16-byte grid
                    const int vecs = static_cast<int>(nBytes / 16);
                    for (int v0 = lane; v0 - lane < vecs; v0 += 4 * 32) {
                        Vec16 q[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (v0 + u * 32 < vecs) q[u] = ld_vec16_stream(row + b0 + static_cast<int64_t>(v0 + u * 32) * 16);
                        }
                        for (uint32_t m = routes; m != 0; m &= m - 1) {
                            uint8_t *p = a.expandXOut + __shfl_sync(0xffffffffu, myRow, __ffs(m) - 1) * rowBytes + b0;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (v0 + u * 32 < vecs) st_vec16(p + static_cast<int64_t>(v0 + u * 32) * 16, q[u]);
                            }
                        }
                    }
                } else {
                    for (uint32_t m = routes; m != 0; m &= m - 1) {
                        uint8_t *p = a.expandXOut + __shfl_sync(0xffffffffu, myRow, __ffs(m) - 1) * rowBytes;
                        if (nBytes > 0) CopyLanes(p + b0, row + b0, nBytes, lane, 32);
                    }
                }
            }
            if (myExpert >= 0 && part == 0) {
                const float wgt = sm.routeWeight[i * K + lane];
                st_vec16(reinterpret_cast<uint8_t *>(a.assistOut) + static_cast<uint64_t>(myRow) * 16,
                         Vec16{static_cast<uint32_t>(comm->rank), static_cast<uint32_t>(t), static_cast<uint32_t>(lane), static_cast<uint32_t>(myExpert)});
                if (a.assistExtOut != nullptr) {
                    *reinterpret_cast<uint2 *>(a.assistExtOut + static_cast<int64_t>(myRow) * 2) = make_uint2(0u, __float_as_uint(wgt));
                }
                if (a.expandScalesOut != nullptr) a.expandScalesOut[myRow] = wgt;
            }
            __syncwarp();
        }
        if (block == G - 1) {                    // the block with the fewest tokens
            for (int e = tid; e < E; e += EP_BLOCK_THREADS) {
                const int upTo = sm.colPrefix[e + 1];
                a.sendCountsOut[e] = upTo;
                a.expertTokenNumsOut[e] = a.tokenNumsType == TileXREp::TILEXR_EP_TOKEN_NUMS_COUNT ? upTo - sm.colPrefix[e] : upTo;
            }
            if (tid == 0 && a.recvTotalOut != nullptr) *a.recvTotalOut = sm.colPrefix[E];
        }
    }
    PerfStageEnd(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC, static_cast<uint64_t>(nRoutes) * rowBytes);
    PerfStageEnd(perf, TILEXR_PERF_KERNEL_TOTAL);
    // All blocks have passed the barrier: none of them reads these words any more.
    if (block == 0 && tid == 0) {
        if (!CLUSTER) doneBlocks[1] = doneBefore + static_cast<uint32_t>(G);
        if (comm->dfx[TILEXR_DFX_FAIL_CODE] == 0) comm->dfx[TILEXR_DFX_RUN_STATUS] = TILEXR_RUN_FINISHED;       // a failure is every block's
        EndLocalLaunch(comm, w);
    }
    if (!CLUSTER) return;
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");       // nobody leaves while its counts may still be read
}

template <int TRANSPORT> __device__ __forceinline__ void GridBody(const EpDispatchArgs &a) { DispatchLocalBody<TRANSPORT, false>(a); }
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchLocalKernel, EpDispatchArgs, GridBody<EP_PLAIN>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchLocalKernelFp8, EpDispatchArgs, GridBody<EP_FP8>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchLocalKernelFp8Round, EpDispatchArgs, GridBody<EP_FP8_ROUND>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchLocalKernelMxfp8, EpDispatchArgs, GridBody<EP_MXFP8>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchLocalKernelInt8, EpDispatchArgs, GridBody<EP_INT8>, EP_BLOCK_THREADS, 2)

template <int TRANSPORT>
__global__ void __launch_bounds__(EP_BLOCK_THREADS, 1) TileXREpDispatchClusterKernel(const __grid_constant__ EpDispatchArgs a)
{
    DispatchLocalBody<TRANSPORT, true>(a);
}

template <int TRANSPORT> const void *ClusterKernel() { return reinterpret_cast<const void *>(&TileXREpDispatchClusterKernel<TRANSPORT>); }

} // namespace

const KernelEntry &EpDispatchLocalKernelEntry(int64_t quantMode, bool round)
{
    if (round) return TileXREpDispatchLocalKernelFp8RoundEntry;
    switch (quantMode) {
        case TileXREp::TILEXR_EP_QUANT_NONE: return TileXREpDispatchLocalKernelEntry;
        case TileXREp::TILEXR_EP_QUANT_FP8_1X128: return TileXREpDispatchLocalKernelFp8Entry;
        case TileXREp::TILEXR_EP_QUANT_MXFP8_E5M2:
        case TileXREp::TILEXR_EP_QUANT_MXFP8_E4M3: return TileXREpDispatchLocalKernelMxfp8Entry;
        default: return TileXREpDispatchLocalKernelInt8Entry;
    }
}

const void *EpDispatchClusterKernel(int64_t quantMode, bool round)
{
    if (round) return ClusterKernel<EP_FP8_ROUND>();
    switch (quantMode) {
        case TileXREp::TILEXR_EP_QUANT_NONE: return ClusterKernel<EP_PLAIN>();
        case TileXREp::TILEXR_EP_QUANT_FP8_1X128: return ClusterKernel<EP_FP8>();
        case TileXREp::TILEXR_EP_QUANT_MXFP8_E5M2:
        case TileXREp::TILEXR_EP_QUANT_MXFP8_E4M3: return ClusterKernel<EP_MXFP8>();
        default: return ClusterKernel<EP_INT8>();
    }
}

size_t EpDispatchLocalSmemBytes(int numExperts, int routesPerBlock)
{
    return static_cast<size_t>(routesPerBlock) * 12 + static_cast<size_t>(numExperts) * 12 + 4 + 32 * 4;
}

} // namespace TileXR
