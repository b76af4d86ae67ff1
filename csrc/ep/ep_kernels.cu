// Expert-parallel dispatch and combine for sm_100a, plus the local hot ops around them
// (routing top-k, block-scaled fp8 quantisation, MXFP8, RMSNorm).
//
// Dispatch, one cooperative kernel per rank:
//   1. every block takes a contiguous range of tokens, routes them (top-k over the gate logits,
//      or reads the given expert ids and masks), and ranks its routes per expert in (token, k)
//      order; per-block expert counts go to a scratch table;
//   2. blocks also add their counts to the rank's totals; the block that finishes last pushes the totals
//      to every peer as epoch-tagged 16-byte units (an all-gather of R x E integers without fence or
//      flag), and a block goes on as soon as the blocks before it have written their counts (no grid
//      barrier).  With everybody's counts each rank computes, for itself as a sender, the exact row at
//      which each of its routes lands in the destination's expert-major / source-major layout: rows are
//      placed at their FINAL position by the sender, the receiver never sorts or compacts;
//   3. a warp per token quantises the row once (fp8 e4m3, one fp32 scale per 128 elements, kept
//      in registers) and stores it to each destination together with its scales and the assist
//      tuple; when the block is done it raises one flag per destination;
//   4. the receiver waits for the flags of every sender block and copies rows, scales and
//      tuples from its window to the output tensors (rows are skipped when the output tensor
//      is registered and was written directly).
// The reference reaches the same layout with worst-case regions per (source, expert) and a
// receiver-side compaction (src/ep/kernels/tilexr_ep_dispatch_memory_kernel.h:666-708,
// 903-1140, 1190-1317); at 4096 tokens x 8 routes that needs gigabytes of window, hence the
// count-first placement here.
//
// Combine: a warp per received row pushes it to slot (token, k) of the source's window and
// raises that slot's flag; a warp per token waits for its K flags and accumulates
// weight_k * row_k in fp32 in k order, then rounds once.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <algorithm>
#include <cstdio>
#include <tuple>
#include <cuda_runtime_api.h>

#include "device/tilexr_data_as_flag.cuh"
#include "device/tilexr_perf_trace.cuh"
#include "device/tilexr_rma.cuh"
#include "device/tilexr_sync.cuh"
#include "device/tilexr_convert.cuh"
#include "ep_device.cuh"
#include "ep_kernels.cuh"
#include "tilexr_ep.h"

namespace TileXR {

using namespace tilexr;

namespace {

__global__ void __launch_bounds__(256) RoutingTopKKernel(const RoutingArgs a)
{
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    const int lane = threadIdx.x & 31;
    if (warp >= a.bs) return;
    float picked;
    RouteToken(a.gateLogits + static_cast<int64_t>(warp) * a.numExperts, a.selectionBias, a.numExperts, a.topK, a.scoreFunc,
               a.renormalize, a.routedScale, lane, a.topkIdsOut + static_cast<int64_t>(warp) * a.topK,
               a.topkWeightsOut + static_cast<int64_t>(warp) * a.topK, &picked);
}

// ---- dispatch ---------------------------------------------------------------------------------------------

struct DispatchSmem {
    int32_t *routeExpert;   // [routesPerBlock]  expert id or -1
    int32_t *routeRank;     // [routesPerBlock]  rank among the block's routes to the same expert
    int32_t *hist;          // [E] routes of this block per expert
    int32_t *blockBase;     // [E] routes of earlier blocks per expert
    int32_t *total;         // [E] routes of all sources per expert
    int32_t *dstRow;        // [E] first row, at the owner, of (expert, this source)
    float *scaleStage;      // [EP_WARPS][64]
    int32_t *colPrefix;     // [E + 1] routes of all sources to the columns before e
};

__device__ __forceinline__ DispatchSmem CarveSmem(uint8_t *base, int numExperts, int routesPerBlock)
{
    DispatchSmem s;
    s.routeExpert = reinterpret_cast<int32_t *>(base);
    s.routeRank = s.routeExpert + routesPerBlock;
    s.hist = s.routeRank + routesPerBlock;
    s.blockBase = s.hist + numExperts;
    s.total = s.blockBase + numExperts;
    s.dstRow = s.total + numExperts;
    s.scaleStage = reinterpret_cast<float *>(s.dstRow + numExperts);
    s.colPrefix = reinterpret_cast<int32_t *>(s.scaleStage + EP_WARPS * 64);
    return s;
}

// out[e] = sum over blocks b in [0, nb) of counts[b * E + e], by all threads of the block.  With E a multiple
// of four a thread adds 16-byte vectors of several rows, so the chain of dependent loads is nb / (threads /
// (E / 4)) long instead of nb.
__device__ void SumBlockCounts(const int32_t *counts, int E, int nb, int32_t *out, int tid, int nThreads)
{
    for (int e = tid; e < E; e += nThreads) out[e] = 0;
    __syncthreads();
    if ((E & 3) == 0) {
        const int vecPerRow = E / 4;
        const int rowsPar = max(1, nThreads / vecPerRow);
        for (int idx = tid; idx < vecPerRow * rowsPar; idx += nThreads) {
            const int col = idx % vecPerRow;
            int4 acc = make_int4(0, 0, 0, 0);
#pragma unroll 4
            for (int b = idx / vecPerRow; b < nb; b += rowsPar) {
                const int4 v = *reinterpret_cast<const int4 *>(counts + static_cast<int64_t>(b) * E + col * 4);
                acc.x += v.x;
                acc.y += v.y;
                acc.z += v.z;
                acc.w += v.w;
            }
            atomicAdd(&out[col * 4 + 0], acc.x);
            atomicAdd(&out[col * 4 + 1], acc.y);
            atomicAdd(&out[col * 4 + 2], acc.z);
            atomicAdd(&out[col * 4 + 3], acc.w);
        }
    } else {
        for (int e = tid; e < E; e += nThreads) {
            int c = 0;
            for (int b = 0; b < nb; ++b) c += counts[static_cast<int64_t>(b) * E + e];
            out[e] = c;
        }
    }
    __syncthreads();
}

// Stage names of the profiler as the EP kernels use them: chunk_total = routing and counting (dispatch) or
// nothing (combine); chunk_barrier = wait for the earlier blocks' counts; post_sync = count exchange and row placement;
// local_input_to_ipc = rows pushed to their destinations; flag_poll_wait = waiting for arrivals;
// peer_ipc_to_output = window to output (dispatch) or the weighted reduction (combine).

template <int TRANSPORT>
__device__ void EpDispatchBody(const EpDispatchArgs &a)
{
    extern __shared__ __align__(16) uint8_t smemRaw[];
    Waiter w;
    bool ok = KernelPrologue(w, a.comm, a.magic, TILEXR_OP_EP_DISPATCH, a.bs, true);
    CommArgs *comm = a.comm;
    const int rank = comm->rank;
    const int R = comm->rankSize;
    const int E = a.numExperts;          // routed experts (what the router chooses from)
    const int C = a.numCols;             // columns of the count tables: shared ranks first, then the routed experts
    const int K = a.topK;
    const int KR = K + a.topo.sharedExperts;   // routes per token: top-k and one per shared expert
    const int G = gridDim.x;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const uint32_t epoch = w.epoch;
    const int routesPerBlock = static_cast<int>(a.tokensPerBlock) * KR;
    // the tables also serve as scratch for the final scan over (local expert, source): moePerRank * R numbers
    DispatchSmem sm = CarveSmem(smemRaw, max(C, a.topo.moePerRank * R), routesPerBlock);
    uint8_t *myHalf = DataHalf(comm, rank, epoch);
    PerfScope perf = PerfInit(tid == 0 ? a.perfTrace : nullptr, static_cast<uint32_t>(rank), blockIdx.x);
    PerfStageBegin(perf, TILEXR_PERF_KERNEL_TOTAL);
    PerfStageBegin(perf, TILEXR_PERF_CHUNK_TOTAL);
    int32_t *blockCounts = reinterpret_cast<int32_t *>(myHalf + a.win.blockCountOff);
    // operator scratch of the rank's control block (tilexr_comm_args.h): a count of the blocks that have finished
    // counting and the rank's totals per column, both back to zero when the launch ends; and one word per
    // block that holds the epoch of the launch whose histogram the block has written (never cleared)
    uint32_t *doneBlocks = reinterpret_cast<uint32_t *>(CtrlWord(comm, rank, TILEXR_CTRL_SCRATCH_WORD + EP_SCRATCH_DONE_WORD));
    uint32_t *totals = reinterpret_cast<uint32_t *>(CtrlWord(comm, rank, TILEXR_CTRL_SCRATCH_WORD + EP_SCRATCH_TOTALS_WORD));
    uint32_t *histReady = reinterpret_cast<uint32_t *>(CtrlWord(comm, rank, TILEXR_CTRL_SCRATCH_WORD + EP_SCRATCH_READY_WORD));
    int32_t *srcBlocks = reinterpret_cast<int32_t *>(sm.scaleStage);       // [R] blocks of each source that raise a flag
    const int units = (C + 1 + 2) / 3;           // 16-byte units of one source's counts: C counts and its block count
    const uint8_t *llMine = LlHalf(comm, rank, epoch);
    __shared__ int sIsLast;
    // whatever becomes of the launch, like the caller's other zeros would have been
    if (blockIdx.x == 0 && tid == 0 && a.laneCountOut != nullptr) *a.laneCountOut = 0;

    const int t0 = min(a.bs, static_cast<int>(blockIdx.x * a.tokensPerBlock));
    const int t1 = min(a.bs, t0 + static_cast<int>(a.tokensPerBlock));
    const int nTok = t1 - t0;
    const int nRoutes = nTok * KR;

    // The block's tokens start on their way to L2 now: memory is idle while the routes are counted.
    {
        const uint8_t *rows = a.x + static_cast<int64_t>(t0) * a.h * a.elemSize;
        const int64_t bytes = static_cast<int64_t>(nTok) * a.h * a.elemSize;
        for (int64_t off = static_cast<int64_t>(tid) * 128; off < bytes; off += static_cast<int64_t>(EP_BLOCK_THREADS) * 128) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(rows + off));
        }
    }

    // ---- 1. route, rank, count (routeExpert holds the COLUMN of a route, -1 when inactive) ---------------
    for (int e = tid; e < C; e += blockDim.x) sm.hist[e] = 0;
    for (int i = warp; i < nTok; i += EP_WARPS) {
        const int t = t0 + i;
        int picked = -1;
        if (a.gateLogits != nullptr) {
            float weight;
            picked = RouteToken(a.gateLogits + static_cast<int64_t>(t) * E, a.selectionBias, E, K, a.scoreFunc, a.renormalize,
                       a.routedScale, lane, a.topkIdsOut + static_cast<int64_t>(t) * K,
                       a.topkWeightsOut + static_cast<int64_t>(t) * K, &weight);
        }
        if (lane < K) {
            int e = a.gateLogits != nullptr ? picked : a.expertIds[static_cast<int64_t>(t) * K + lane];
            if (e < 0 || e >= E) e = -1;
            if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_TOKEN && a.activeMask[t] == 0) e = -1;
            if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_EXPERT && a.activeMask[static_cast<int64_t>(t) * K + lane] == 0) e = -1;
            sm.routeExpert[i * KR + lane] = e >= 0 ? a.topo.sharedRanks + e : -1;
            if (a.gateLogits == nullptr && a.topkIdsOut != nullptr) a.topkIdsOut[static_cast<int64_t>(t) * K + lane] = e;
        } else if (lane < KR) {
            // every active token also goes to its copy of each shared expert
            const bool active = !(a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_TOKEN && a.activeMask[t] == 0);
            sm.routeExpert[i * KR + lane] = active ? EpSharedCol(a.topo, rank, lane - K) : -1;
        }
    }
    __syncthreads();
    if (warp == 0) RankBlockRoutes(nRoutes, sm.routeExpert, sm.routeRank, sm.hist, lane);
    __syncthreads();
    for (int e = tid; e < C; e += blockDim.x) {
        const int hcount = sm.hist[e];
        blockCounts[static_cast<int64_t>(blockIdx.x) * C + e] = hcount;
        if (hcount != 0) atomicAdd(&totals[e], static_cast<uint32_t>(hcount));
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        st_release_gpu_u32(&histReady[blockIdx.x], epoch);
        sIsLast = atom_add_acq_rel_gpu_u32(doneBlocks, 1u) == static_cast<uint32_t>(G) - 1u ? 1 : 0;
    }
    __syncthreads();
    PerfStageEnd(perf, TILEXR_PERF_CHUNK_TOTAL);
    PerfStageBegin(perf, TILEXR_PERF_POST_SYNC);

    // ---- 2. publish this rank's counts, learn everybody's ----------------------------------------------
    // The block that finishes counting last has the rank's totals in front of it and sends them to every
    // peer as self-validating 16-byte units (three counts and the epoch): no fence, no flag, one NVLink
    // crossing.  Nobody waits at a barrier: a block only needs the histograms of the blocks before it.
    if (ok && sIsLast != 0) {
        for (int u = tid; u < units; u += blockDim.x) {
            uint32_t v[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int idx = u * 3 + q;
                v[q] = idx < C ? __ldcg(&totals[idx]) : (idx == C ? static_cast<uint32_t>(G) : 0u);
            }
            for (int i = 0; i < R; ++i) {
                const int peer = (rank + i) % R;
                Ll16SendUnit(LlHalf(comm, peer, epoch) + (static_cast<uint64_t>(rank) * units + u) * LL16_UNIT_BYTES, v[0], v[1], v[2], epoch);
            }
        }
    }
    PerfStageBegin(perf, TILEXR_PERF_CHUNK_BARRIER);
    {
        bool got = true;
        for (int b = tid; ok && got && b < static_cast<int>(blockIdx.x); b += blockDim.x) {
            uint32_t polls = 0;
            while (ld_acquire_gpu_u32(&histReady[b]) != epoch) {
                if ((++polls & 63u) == 0) {
                    const uint64_t t = now_ns();
                    if (w.deadline == 0) {
                        w.deadline = t + w.args->waitTimeoutNs;
                    } else if (t > w.deadline || AbortRaised(w)) {
                        RaiseFailure(w, TILEXR_DEV_GRID_BARRIER_TIMEOUT, rank, b, epoch, histReady[b]);
                        got = false;
                        break;
                    }
                }
                spin_pause();
            }
        }
        ok = BlockBroadcastOk(got) && ok;
    }
    PerfStageEnd(perf, TILEXR_PERF_CHUNK_BARRIER);
    SumBlockCounts(blockCounts, C, ok ? static_cast<int>(blockIdx.x) : 0, sm.blockBase, tid, blockDim.x);
    for (int e = tid; e < C; e += blockDim.x) {
        sm.total[e] = 0;
        sm.hist[e] = 0;       // from here on: routes of lower ranks to column e
    }
    __syncthreads();
    {
        bool got = true;
        for (int u = tid; ok && got && u < R * units; u += blockDim.x) {
            const int s = u / units;
            const int j = u - s * units;
            Vec16 v;
            got = Ll16WaitUnit(w, llMine + static_cast<uint64_t>(u) * LL16_UNIT_BYTES, s, u, &v);
            if (!got) break;
            const uint32_t vals[3] = {v.x, v.y, v.z};
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const int idx = j * 3 + q;
                if (idx < C) {
                    if (vals[q] != 0) {
                        atomicAdd(&sm.total[idx], static_cast<int32_t>(vals[q]));
                        if (s < rank) atomicAdd(&sm.hist[idx], static_cast<int32_t>(vals[q]));
                    }
                } else if (idx == C) {
                    srcBlocks[s] = static_cast<int32_t>(vals[q]);
                }
            }
        }
        ok = BlockBroadcastOk(got) && ok;
    }
    if (ok) {
        // prefix sums of the totals: warps scan 32 columns each, then every warp scans the (at most 32) sums of those
        const int groups32 = (C + 31) / 32;
        int32_t *groupSum = reinterpret_cast<int32_t *>(sm.scaleStage) + EP_WARPS * 32;
        for (int c = warp; c < groups32; c += EP_WARPS) {
            int v = c * 32 + lane < C ? sm.total[c * 32 + lane] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            if (c * 32 + lane < C) sm.colPrefix[c * 32 + lane + 1] = v;
            if (lane == 31) groupSum[c] = v;
        }
        __syncthreads();
        {
            const int own = lane < groups32 ? groupSum[lane] : 0;
            int v = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += u;
            }
            for (int c = warp; c < groups32; c += EP_WARPS) {
                const int before = __shfl_sync(0xffffffffu, v - own, c);
                if (c * 32 + lane < C) sm.colPrefix[c * 32 + lane + 1] += before;
            }
            if (tid == 0) sm.colPrefix[0] = 0;
        }
        __syncthreads();
        for (int e = tid; e < C; e += blockDim.x) {
            sm.dstRow[e] = sm.hist[e] + sm.colPrefix[e] - sm.colPrefix[EpRankFirstCol(a.topo, EpColRank(a.topo, e))];
        }
        // Every rank sees the same counts, so every rank reaches the same verdict on overflow.
        bool fits = true;
        if (tid < R) {
            const int firstCol = EpRankFirstCol(a.topo, tid);
            const int64_t rows = sm.colPrefix[firstCol + EpRankCols(a.topo, tid)] - sm.colPrefix[firstCol];
            fits = rows <= static_cast<int64_t>(a.maxRecvRows);
            if (!fits) RaiseFailure(w, TILEXR_DEV_BAD_ARGUMENT, tid, 0, a.maxRecvRows, static_cast<uint64_t>(rows));
        }
        ok = BlockBroadcastOk(fits);
    }

    PerfStageEnd(perf, TILEXR_PERF_POST_SYNC);

    // ---- 3. send ----------------------------------------------------------------------------------------
    PerfStageBegin(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC);
    if (ok) {
        const bool bf16 = a.isBf16 != 0;
        constexpr bool mx = TRANSPORT == EP_MXFP8;
        const bool mxE5m2 = a.quantMode == TileXREp::TILEXR_EP_QUANT_MXFP8_E5M2;
        constexpr bool quant = mx || TRANSPORT == EP_FP8;
        const bool int8Dynamic = a.quantMode == TileXREp::TILEXR_EP_QUANT_DYNAMIC_INT8;
        constexpr bool int8Mode = TRANSPORT == EP_INT8;
        const int chunks = a.h / 16;             // 16 elements per lane and iteration (fp8 paths)
        const int iters = (chunks + 31) / 32;
        // A block with few tokens (small batches) cuts every token into column ranges for several warps.
        const int parts = nTok > 0 ? max(1, min(min(8, iters), static_cast<int>(EP_WARPS) / nTok)) : 1;
        // where the scales of row `rr` go at the destination whose window half is `half`
        auto scaleRow = [&](unsigned long long half, uint32_t rr) {
            return reinterpret_cast<uint8_t *>(half) + a.win.scalesOff + static_cast<uint64_t>(rr) * a.win.scaleRowBytes;
        };
        for (int item = warp; item < nTok * parts; item += EP_WARPS) {
            const int i = item / parts;
            const int part = item % parts;
            const int t = t0 + i;
            const uint8_t *row = a.x + static_cast<int64_t>(t) * a.h * a.elemSize;
            // lane k owns route k of this token: where its row, scales and tuple go
            unsigned long long myPayload = 0, myHalf = 0;
            uint32_t myRow = 0;
            int myExpert = -1;
            if (lane < KR) {
                const int e = sm.routeExpert[i * KR + lane];
                if (e >= 0) {
                    const int dst = EpColRank(a.topo, e);
                    myRow = static_cast<uint32_t>(sm.dstRow[e] + sm.blockBase[e] + sm.routeRank[i * KR + lane]);
                    uint8_t *half = DataHalf(comm, dst, epoch);
                    // rows for this rank's own experts go to the output directly (the receive step skips their payload)
                    uint8_t *payload = dst == rank && a.directOwn != 0
                                           ? a.expandXOut + static_cast<uint64_t>(myRow) * a.win.rowBytes
                                       : a.zeroCopy
                                           ? comm->registryPtr->regions[a.outHandle].peerBase[dst] + a.outOffset +
                                                 static_cast<uint64_t>(myRow) * a.win.rowBytes
                                           : half + a.win.payloadOff + static_cast<uint64_t>(myRow) * a.win.rowBytes;
                    myPayload = reinterpret_cast<unsigned long long>(payload);
                    myHalf = reinterpret_cast<unsigned long long>(half);
                    myExpert = e;
                }
            }
            if (lane < KR && a.routeRowsOut != nullptr && part == 0) {
                a.routeRowsOut[static_cast<int64_t>(t) * KR + lane] = myExpert >= 0 ? static_cast<int32_t>(myRow) : -1;
            }
            const uint32_t routes = __ballot_sync(0xffffffffu, myExpert >= 0);
            if (routes == 0) continue;
            // Routes of this token to one remote rank form a group: the lowest k (the head) carries the
            // payload, the others only their tuple, and every member links to the next one.
            const int myDst = myExpert >= 0 ? EpColRank(a.topo, myExpert) : -1;
            uint32_t myLink = 0;
            if (a.dedup != 0) {
                bool follower = false;
                for (int j = 0; j < KR; ++j) {
                    const int dj = __shfl_sync(0xffffffffu, myDst, j);
                    const uint32_t rj = __shfl_sync(0xffffffffu, myRow, j);
                    if (dj >= 0 && dj == myDst && myDst != rank) {
                        if (j < lane) follower = true;
                        else if (j > lane && myLink == 0) myLink = rj + 1;
                    }
                }
                if (follower) myLink |= EP_LINK_FOLLOWER;
            }
            const uint32_t payloadRoutes = __ballot_sync(0xffffffffu, myExpert >= 0 && (myLink & EP_LINK_FOLLOWER) == 0);
            if (int8Mode) {
                // int8 with optional per-expert smoothing scales: every route is quantised for its own expert.
                // dynamic: one pass for the row's amax (scale = amax / 127, stored beside the row), one to convert;
                // static: the caller's scales already map into int8 range.
                uint32_t m = payloadRoutes;
                while (m != 0) {
                    const int k = __ffs(m) - 1;
                    m &= m - 1;
                    uint8_t *p = reinterpret_cast<uint8_t *>(__shfl_sync(0xffffffffu, myPayload, k));
                    const unsigned long long half = __shfl_sync(0xffffffffu, myHalf, k);
                    const uint32_t rr = __shfl_sync(0xffffffffu, myRow, k);
                    const int e = __shfl_sync(0xffffffffu, myExpert, k);
                    const float *sc = (a.quantScales != nullptr && e >= a.topo.sharedRanks)
                                          ? a.quantScales + static_cast<int64_t>(e - a.topo.sharedRanks) * a.h : nullptr;
                    float inv = 1.0f;
                    if (int8Dynamic) {
                        const float amax = Int8RowAmax(row, sc, chunks, bf16, lane);
                        if (amax > 0.f) inv = 127.0f / amax;
                        if (part == 0 && lane == 0) {
                            const float scale = amax > 0.f ? amax / 127.0f : 1.0f;
                            st_vec16(scaleRow(half, rr), Vec16{__float_as_uint(scale), 0u, 0u, 0u});     // a 16-byte cell in the window
                        }
                    }
                    Int8RowStore(row, sc, inv, chunks, bf16, part, parts, lane, p);
                }
            } else if (quant) {
                // each 512-element chunk is quantised once and stored to every destination right away:
                // nothing row-sized lives in registers, so two blocks fit on an SM
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
                    // this iteration's 16 bytes of the scale row: lane k stores them for route k
                    Vec16 sv;
                    const Vec16 q = mx ? QuantMx16(f, mxE5m2, lane, &sv) : QuantFp8Block16(f, &sv);
                    if ((payloadRoutes >> lane) & 1u) st_vec16(scaleRow(myHalf, myRow) + it * 16, sv);
                    uint32_t m = payloadRoutes;
                    while (m != 0) {
                        const int k = __ffs(m) - 1;
                        m &= m - 1;
                        uint8_t *p = reinterpret_cast<uint8_t *>(__shfl_sync(0xffffffffu, myPayload, k));
                        if (c < chunks) st_vec16(p + static_cast<int64_t>(c) * 16, q);
                    }
                }
            } else {
                const uint64_t perPart = ((a.win.rowBytes + parts - 1) / parts + 511) & ~511ull;
                const uint64_t b0 = min(static_cast<uint64_t>(a.win.rowBytes), perPart * part);
                const uint64_t nBytes = min(static_cast<uint64_t>(a.win.rowBytes) - b0, perPart);
                const bool odd = __any_sync(0xffffffffu, ((myPayload | reinterpret_cast<unsigned long long>(row)) & 15ull) != 0) || (nBytes & 15ull) != 0;
                if (!odd) {
                    // the part is fetched once and stored to every destination (one copy per destination fetched it again each
                    // time, a round trip per 2 KB: 1009 x 4096, top-6, 10 us of the launch)
                    const int vecs = static_cast<int>(nBytes / 16);
                    for (int v0 = lane; v0 - lane < vecs; v0 += 4 * 32) {
                        Vec16 q[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (v0 + u * 32 < vecs) q[u] = ld_vec16_stream(row + b0 + static_cast<int64_t>(v0 + u * 32) * 16);
                        }
                        uint32_t m = payloadRoutes;
                        while (m != 0) {
                            const int k = __ffs(m) - 1;
                            m &= m - 1;
                            uint8_t *p = reinterpret_cast<uint8_t *>(__shfl_sync(0xffffffffu, myPayload, k)) + b0;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                if (v0 + u * 32 < vecs) st_vec16(p + static_cast<int64_t>(v0 + u * 32) * 16, q[u]);
                            }
                        }
                    }
                } else {
                    uint32_t m = payloadRoutes;
                    while (m != 0) {
                        const int k = __ffs(m) - 1;
                        m &= m - 1;
                        uint8_t *p = reinterpret_cast<uint8_t *>(__shfl_sync(0xffffffffu, myPayload, k));
                        if (nBytes > 0) CopyLanes(p + b0, row + b0, nBytes, lane, 32);
                    }
                }
            }
            if (myExpert >= 0 && part == 0) {
                st_vec16(reinterpret_cast<uint8_t *>(myHalf) + a.win.assistOff + static_cast<uint64_t>(myRow) * 16,
                         Vec16{static_cast<uint32_t>(rank), static_cast<uint32_t>(t), static_cast<uint32_t>(lane),
                               static_cast<uint32_t>(lane < K ? myExpert - a.topo.sharedRanks : lane - K)});   // routed expert id, or shared expert id
                const int64_t route = static_cast<int64_t>(t) * K + lane;
                const float wgt = lane >= K ? 1.0f
                                  : a.gateLogits != nullptr ? a.topkWeightsOut[route]
                                                            : (a.expertScales != nullptr ? a.expertScales[route] : 1.0f);
                *reinterpret_cast<uint2 *>(reinterpret_cast<uint8_t *>(myHalf) + a.win.extOff + static_cast<uint64_t>(myRow) * 8) =
                    make_uint2(myLink, __float_as_uint(wgt));
            }
            __syncwarp();
        }
    }
    __syncthreads();
    if (ok && tid < R) {
        SetFlag(FlagSlot(comm, tid, TILEXR_FLAG_OP_BASE + static_cast<int64_t>(rank) * TILEXR_FLAGS_PER_PAIR + blockIdx.x), epoch, 1);
    }
    PerfStageEnd(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC, static_cast<uint64_t>(nRoutes) * a.win.rowBytes);

    // ---- 4. receive ---------------------------------------------------------------------------------------
    PerfStageBegin(perf, TILEXR_PERF_FLAG_POLL_WAIT);
    {
        // every thread polls its share of the (source, block) flags; a source's block count came with its counts
        bool got = true;
        if (ok) {
            for (int s = 0; s < R && got; ++s) {
                const int64_t base = TILEXR_FLAG_OP_BASE + static_cast<int64_t>(s) * TILEXR_FLAGS_PER_PAIR;
                const int blocksOfS = min(srcBlocks[s], static_cast<int>(EP_COUNT_FLAG_SLOT));
                for (int b = tid; b < blocksOfS && got; b += blockDim.x) {
                    got = WaitFlagGE(w, FlagSlot(comm, rank, base + b), 1, s, base + b);
                }
            }
        }
        ok = BlockBroadcastOk(got) && ok;
    }
    PerfStageEnd(perf, TILEXR_PERF_FLAG_POLL_WAIT);
    PerfStageBegin(perf, TILEXR_PERF_PEER_IPC_TO_OUTPUT);
    if (ok) {
        const int firstLocal = EpRankFirstCol(a.topo, rank);
        const int localCols = EpRankCols(a.topo, rank);
        const int64_t rows = sm.colPrefix[firstLocal + localCols] - sm.colPrefix[firstLocal];
        // Rows are dealt out to blocks in chunks of one row per thread.  Per chunk: (a) a thread per row copies
        // the tuple, link and weight and notes the head rows that have followers; (b) a thread per 16 bytes
        // copies the scales of the rows that arrived with a payload; (c) without zero-copy a warp per row moves
        // the payload out of the window; (d) warps take the noted head rows in turn and fill their followers.
        const bool quantOut = a.win.scaleRowBytes != 0 && a.dynamicScalesOut != nullptr;
        const bool scalarScale = a.quantMode == TileXREp::TILEXR_EP_QUANT_DYNAMIC_INT8;     // one fp32 per row in the output
        const uint8_t *winPayload = myHalf + a.win.payloadOff;
        const uint8_t *winScales = myHalf + a.win.scalesOff;
        const uint8_t *winExt = myHalf + a.win.extOff;
        __shared__ int32_t sHead[EP_BLOCK_THREADS];
        __shared__ int sHeadCount;
        const int scaleVecsPerRow = static_cast<int>(a.win.scaleRowBytes / 16);
        // a chunk is as small as it takes to give every block rows (32 at least), and one row per thread at most
        const int64_t chunk = min(static_cast<int64_t>(EP_BLOCK_THREADS), max(static_cast<int64_t>(32), static_cast<int64_t>(((rows + G - 1) / G + 31) & ~static_cast<int64_t>(31))));
        for (int64_t base = static_cast<int64_t>(blockIdx.x) * chunk; base < rows; base += static_cast<int64_t>(G) * chunk) {
            const int chunkRows = static_cast<int>(min(chunk, rows - base));
            if (tid == 0) sHeadCount = 0;
            __syncthreads();
            if (tid < chunkRows) {
                const int64_t r = base + tid;
                const uint2 ext = *reinterpret_cast<const uint2 *>(winExt + r * 8);
                st_vec16(reinterpret_cast<uint8_t *>(a.assistOut) + r * 16, ld_vec16(myHalf + a.win.assistOff + r * 16));
                if (a.assistExtOut != nullptr) *reinterpret_cast<uint2 *>(a.assistExtOut + r * 2) = ext;
                if (a.expandScalesOut != nullptr) a.expandScalesOut[r] = __uint_as_float(ext.y);
                if (a.dedup != 0 && (ext.x & EP_LINK_FOLLOWER) == 0 && (ext.x & EP_LINK_NEXT_MASK) != 0) {
                    sHead[atomicAdd(&sHeadCount, 1)] = tid;
                }
            }
            if (quantOut) {
                for (int idx = tid; idx < chunkRows * scaleVecsPerRow; idx += EP_BLOCK_THREADS) {
                    const int64_t r = base + idx / scaleVecsPerRow;
                    const int v = idx % scaleVecsPerRow;
                    if ((reinterpret_cast<const uint2 *>(winExt + r * 8)->x & EP_LINK_FOLLOWER) != 0) continue;
                    if (scalarScale) {
                        a.dynamicScalesOut[r] = *reinterpret_cast<const float *>(winScales + r * a.win.scaleRowBytes);
                        continue;
                    }
                    st_vec16(reinterpret_cast<uint8_t *>(a.dynamicScalesOut) + r * a.win.scaleRowBytes + v * 16,
                             ld_vec16(winScales + r * a.win.scaleRowBytes + v * 16));
                }
            }
            if (!a.zeroCopy) {
                for (int i = warp; i < chunkRows; i += EP_WARPS) {
                    const int64_t r = base + i;
                    if ((reinterpret_cast<const uint2 *>(winExt + r * 8)->x & EP_LINK_FOLLOWER) != 0) continue;
                    if (a.directOwn != 0 && *reinterpret_cast<const int32_t *>(myHalf + a.win.assistOff + r * 16) == rank) continue;   // already there
                    CopyLanes(a.expandXOut + r * a.win.rowBytes, winPayload + r * a.win.rowBytes, a.win.rowBytes, lane, 32);
                }
            }
            __syncthreads();
            const int heads = sHeadCount;
            for (int u = warp; u < heads; u += EP_WARPS) {
                const int64_t r = base + sHead[u];
                const uint8_t *src = a.zeroCopy ? a.expandXOut + r * a.win.rowBytes : winPayload + r * a.win.rowBytes;
                // lane j keeps follower j of the chain; the head row is then read once and stored to all of them
                int64_t myFollower = -1;
                int followers = 0;
                uint32_t next = reinterpret_cast<const uint2 *>(winExt + r * 8)->x & EP_LINK_NEXT_MASK;
                for (int hop = 0; next != 0 && hop < KR; ++hop) {
                    const int64_t f = static_cast<int64_t>(next) - 1;
                    if (f >= static_cast<int64_t>(a.maxRecvRows)) break;
                    if (lane == followers) myFollower = f;
                    ++followers;
                    next = reinterpret_cast<const uint2 *>(winExt + f * 8)->x & EP_LINK_NEXT_MASK;
                }
                const int rowVecs16 = a.directOwn != 0 ? static_cast<int>(a.win.rowBytes / 16) : 0;     // an output off the 16-byte grid takes single bytes
                for (int v0 = 0; v0 < rowVecs16; v0 += 128) {
                    Vec16 q[4];
#pragma unroll
                    for (int k4 = 0; k4 < 4; ++k4) {
                        const int v = v0 + k4 * 32 + lane;
                        if (v < rowVecs16) q[k4] = ld_vec16_stream(src + static_cast<int64_t>(v) * 16);
                    }
                    for (int j = 0; j < followers; ++j) {
                        uint8_t *dst = a.expandXOut + __shfl_sync(0xffffffffu, myFollower, j) * a.win.rowBytes;
#pragma unroll
                        for (int k4 = 0; k4 < 4; ++k4) {
                            const int v = v0 + k4 * 32 + lane;
                            if (v < rowVecs16) st_vec16(dst + static_cast<int64_t>(v) * 16, q[k4]);
                        }
                    }
                }
                for (int j = 0; j < followers; ++j) {
                    uint8_t *dst = a.expandXOut + __shfl_sync(0xffffffffu, myFollower, j) * a.win.rowBytes;
                    for (uint32_t i = static_cast<uint32_t>(rowVecs16) * 16 + lane; i < a.win.rowBytes; i += 32) dst[i] = src[i];
                }
                for (int j = 0; j < followers; ++j) {
                    const int64_t f = __shfl_sync(0xffffffffu, myFollower, j);
                    if (quantOut && scalarScale) {
                        if (lane == 0) a.dynamicScalesOut[f] = *reinterpret_cast<const float *>(winScales + r * a.win.scaleRowBytes);
                    } else if (quantOut) {
                        CopyLanes(reinterpret_cast<uint8_t *>(a.dynamicScalesOut) + f * a.win.scaleRowBytes,
                                  winScales + r * a.win.scaleRowBytes, a.win.scaleRowBytes, lane, 32);
                    }
                }
            }
            __syncthreads();
        }
        if (blockIdx.x == 0) {
            // cumulative counts in (local expert, source) order: an inclusive scan of E_local * R numbers
            const int n = localCols * R;
            __syncthreads();
            for (int i = tid; i < n; i += blockDim.x) {
                // count of source i % R for local column i / R, out of that source's units (all seen to be complete above)
                const int idx = firstLocal + i / R;
                sm.hist[i] = static_cast<int32_t>(reinterpret_cast<const uint32_t *>(
                    llMine + (static_cast<uint64_t>(i % R) * units + idx / 3) * LL16_UNIT_BYTES)[idx % 3]);
            }
            __syncthreads();
            if (warp == 0) {
                int carry = 0;
                for (int base = 0; base < n; base += 32) {
                    int v = base + lane < n ? sm.hist[base + lane] : 0;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int u = __shfl_up_sync(0xffffffffu, v, o);
                        if (lane >= o) v += u;
                    }
                    v += carry;
                    if (base + lane < n) sm.hist[base + lane] = v;
                    carry = __shfl_sync(0xffffffffu, v, 31);
                }
            }
            __syncthreads();
            for (int i = tid; i < n; i += blockDim.x) a.sendCountsOut[i] = sm.hist[i];
            for (int le = tid; le < localCols; le += blockDim.x) {
                a.expertTokenNumsOut[le] = a.tokenNumsType == TileXREp::TILEXR_EP_TOKEN_NUMS_COUNT
                                               ? static_cast<int64_t>(sm.total[firstLocal + le])
                                               : static_cast<int64_t>(sm.hist[le * R + R - 1]);
            }
            if (tid == 0 && a.recvTotalOut != nullptr) *a.recvTotalOut = n > 0 ? sm.hist[n - 1] : 0;
        }
    }
    PerfStageEnd(perf, TILEXR_PERF_PEER_IPC_TO_OUTPUT);
    PerfStageEnd(perf, TILEXR_PERF_KERNEL_TOTAL);
    KernelEpilogue(w, ok, EP_SCRATCH_TOTALS_WORD + (C + 1) / 2);
}

// ---- combine -----------------------------------------------------------------------------------------------
//
// Work is handed out by two cursors in the rank's control block, so that no warp idles while another still has
// a queue (rows differ a lot: local rows are skipped, followers are folded into their head, heads sum a chain).
//
//   send items    (bucket, chunk of rows, column part): the warp reads the tuples of the chunk's rows, keeps the
//                 rows that must travel and whose token lies in `bucket`, and sends that column part of each.
//                 Buckets are ranges of the SOURCE's token index, walked in increasing order by every rank, so a
//                 token's slots arrive from all ranks at about the same time and in token order;
//   reduce items  (token, column part) in increasing token order: wait for the part's slot flags, sum.
//
// The last `reducerBlocks` blocks take reduce items from the start, the others first send and then join: the
// reduction of the early buckets overlaps the transfer of the later ones, and after the last row has landed
// only the last bucket is left to sum.  Every (row, part) has a flag of its own, raised by the sending warp.

__device__ __forceinline__ uint32_t TakeItem(uint32_t *cursor, int lane)
{
    uint32_t it = 0;
    if (lane == 0) it = atomicAdd(cursor, 1u);
    return __shfl_sync(0xffffffffu, it, 0);
}

// Sends column part `part` of row `r` to slot `slot` of rank `src` and raises the part's flag there.  A head row
// of a group is replaced by the gate-weighted fp32 sum of the group's rows (one rounding).  Called by a whole warp.
__device__ __forceinline__ void CombineSendPart(const EpCombineArgs &a, CommArgs *comm, uint32_t epoch, int64_t r, int64_t rows,
                                                int src, int64_t slot, uint32_t link, uint32_t weightBits, uint32_t part, int lane)
{
    const bool bf16 = a.isBf16 != 0;
    const int KR = a.topK + a.topo.sharedExperts;
    const int rowVecs = a.rowBytes / 16;
    const int vBegin = static_cast<int>(part) * static_cast<int>(a.partVecs);
    const int vEnd = min(rowVecs, vBegin + static_cast<int>(a.partVecs));
    uint8_t *dst = DataHalf(comm, src, epoch) + slot * a.rowBytes;
    if ((link & EP_LINK_NEXT_MASK) == 0) {
        // eight 16-byte vectors in flight per lane: under an all-to-all of eight ranks a store takes several
        // microseconds to be acknowledged, and the warps on an SM must cover that with bytes in flight
        const uint8_t *src = a.expertOut + r * a.rowBytes;
        int v = vBegin + lane;
        for (; v + 7 * 32 < vEnd; v += 8 * 32) {
            Vec16 q[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) q[u] = ld_vec16_stream(src + static_cast<int64_t>(v + u * 32) * 16);
#pragma unroll
            for (int u = 0; u < 8; ++u) st_vec16(dst + static_cast<int64_t>(v + u * 32) * 16, q[u]);
        }
        // the rest of the row (fewer than eight vectors per lane) in rounds of four with the missing ones switched off;
        // one vector at a time it would cost a round trip each
        for (; v < vEnd; v += 4 * 32) {
            Vec16 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (v + u * 32 < vEnd) q[u] = ld_vec16_stream(src + static_cast<int64_t>(v + u * 32) * 16);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (v + u * 32 < vEnd) st_vec16(dst + static_cast<int64_t>(v + u * 32) * 16, q[u]);
            }
        }
    } else {
        // The rows of this token on this rank, in k order, times their gate weights: lane i keeps member i of
        // the chain, then every 16-byte column is summed in fp32 and rounded once.
        int64_t memberRow = -1;
        float memberW = 0.f;
        int members = 0;
        int64_t cur = r;
        uint2 e2 = make_uint2(link, weightBits);
        while (members < KR) {
            if (lane == members) {
                memberRow = cur;
                memberW = __uint_as_float(e2.y);
            }
            ++members;
            const uint32_t next = e2.x & EP_LINK_NEXT_MASK;
            if (next == 0 || static_cast<int64_t>(next) - 1 >= rows) break;
            cur = static_cast<int64_t>(next) - 1;
            e2 = *reinterpret_cast<const uint2 *>(a.assistExt + cur * 2);
        }
        for (int v0 = vBegin; v0 < vEnd; v0 += 32) {
            const int v = v0 + lane;
            float acc[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = 0.f;
            // the columns of four members are fetched together, then added in k order
            for (int i0 = 0; i0 < members; i0 += 4) {
                Vec16 q[4];
                float mw[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int64_t mr = __shfl_sync(0xffffffffu, memberRow, (i0 + i) & 31);
                    mw[i] = __shfl_sync(0xffffffffu, memberW, (i0 + i) & 31);
                    q[i] = Vec16{0u, 0u, 0u, 0u};
                    if (i0 + i < members && v < vEnd) q[i] = ld_vec16_stream(a.expertOut + mr * a.rowBytes + v * 16);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (i0 + i < members) {
                        float f[8];
                        Unpack8(q[i], bf16, f);
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[j] = fmaf(mw[i], f[j], acc[j]);
                    }
                }
            }
            if (v < vEnd) st_vec16(dst + v * 16, Pack8(acc, bf16));
        }
    }
    // every lane's stores of this part are ordered before the flag by the warp barrier and the release
    __syncwarp();
    if (lane == 0) SetFlag(FlagSlot(comm, src, TILEXR_FLAG_SLOT_BASE + slot * a.parts + part), epoch, 1);
}

__device__ void EpCombineBody(const EpCombineArgs &a)
{
    Waiter w;
    bool ok = KernelPrologue(w, a.comm, a.magic, TILEXR_OP_EP_COMBINE, a.bs, true);
    CommArgs *comm = a.comm;
    const int rank = comm->rank;
    const int K = a.topK;
    const int KR = K + a.topo.sharedExperts;     // slots per token: top-k routes and one per shared expert
    const int lane = threadIdx.x & 31;
    const uint32_t epoch = w.epoch;
    const bool bf16 = a.isBf16 != 0;
    const uint32_t P = a.parts;
    const int rowVecs = a.rowBytes / 16;
    const int partVecs = a.partVecs;
    uint32_t *cursors = reinterpret_cast<uint32_t *>(CtrlWord(comm, rank, TILEXR_CTRL_SCRATCH_WORD));
    PerfScope perf = PerfInit(threadIdx.x == 0 ? a.perfTrace : nullptr, static_cast<uint32_t>(rank), blockIdx.x);
    PerfStageBegin(perf, TILEXR_PERF_KERNEL_TOTAL);

    if (ok) {
        const int64_t rows = a.sendCounts[a.sendCountEntries - 1];
        // Rows of this rank's own tokens stay where they are when the reducer knows their row (direct), and the
        // followers of a group are summed into their head's row.
        const bool direct = a.routeRows != nullptr && a.expertIds != nullptr;
        const bool sender = blockIdx.x + a.reducerBlocks < gridDim.x;
        // What a lane learns about row r: does it travel, where to, which bucket of the source's tokens.
        auto classify = [&](int64_t r, int &src, int64_t &slot, uint2 &ext, uint32_t &bucket) -> bool {
            const Vec16 tuple = ld_vec16(a.assist + r * 4);
            src = static_cast<int>(tuple.x);
            slot = static_cast<int64_t>(tuple.y) * KR + tuple.z;
            bucket = min(tuple.y / a.bucketTokens, a.buckets - 1u);
            bool send = src >= 0 && src < comm->rankSize && tuple.y < static_cast<uint32_t>(a.bs) && tuple.z < static_cast<uint32_t>(KR);
            if (direct && src == rank) send = false;
            if (send && a.dedup != 0) {
                ext = *reinterpret_cast<const uint2 *>(a.assistExt + r * 2);
                if ((ext.x & EP_LINK_FOLLOWER) != 0) send = false;
            }
            return send;
        };
        const uint32_t senders = gridDim.x - a.reducerBlocks;
        const bool sorted = a.buckets > 1 && rows <= static_cast<int64_t>(a.listCap);
        if (sender && sorted) {
            PerfStageBegin(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC);
            // Rows in a (local expert, source) segment are in token order, so consecutive rows share a bucket:
            // the rows that travel are first sorted by bucket into lists (positions by atomics, order within a
            // bucket does not matter), then one cursor walks the lists bucket after bucket, a row part per item.
            uint32_t *bucketCount = cursors + 2 * EP_SCRATCH_BUCKET_WORD;
            int32_t *lists = reinterpret_cast<int32_t *>(DataHalf(comm, rank, epoch) + a.listOff);
            const int64_t gw = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
            const int64_t nw = static_cast<int64_t>(senders) * (blockDim.x >> 5);
            for (int64_t base = gw * 32; base < rows; base += nw * 32) {
                const int64_t r = base + lane;
                int src = -1;
                int64_t slot = 0;
                uint2 ext = make_uint2(0u, 0u);
                uint32_t bucket = 0;
                const bool send = r < rows && classify(r, src, slot, ext, bucket);
                uint32_t left = __ballot_sync(0xffffffffu, send);
                while (left != 0) {
                    const uint32_t bb = __shfl_sync(0xffffffffu, bucket, __ffs(left) - 1);
                    const uint32_t m = __ballot_sync(0xffffffffu, send && bucket == bb);
                    uint32_t pos = 0;
                    if (lane == 0) pos = atomicAdd(&bucketCount[bb], static_cast<uint32_t>(__popc(m)));
                    pos = __shfl_sync(0xffffffffu, pos, 0);
                    if (send && bucket == bb) lists[static_cast<uint64_t>(bb) * a.listCap + pos + __popc(m & ((1u << lane) - 1u))] = static_cast<int32_t>(r);
                    left &= ~m;
                }
            }
            __syncthreads();
            {
                bool got = true;
                if (threadIdx.x == 0) {
                    __threadfence();
                    got = GridBarrierThread0(w, 1, senders);
                }
                ok = BlockBroadcastOk(got);
            }
            if (ok) {
                uint32_t incl = lane < static_cast<int>(a.buckets) ? __ldcg(&bucketCount[lane]) : 0u;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                const uint32_t nItems = __shfl_sync(0xffffffffu, incl, 31) * P;
                for (;;) {
                    const uint32_t it = TakeItem(&cursors[0], lane);
                    if (it >= nItems) break;
                    const uint32_t i = it / P;
                    const uint32_t part = it - i * P;
                    const int b = __popc(__ballot_sync(0xffffffffu, lane < static_cast<int>(a.buckets) && incl <= i));
                    const uint32_t before = b > 0 ? __shfl_sync(0xffffffffu, incl, b - 1) : 0u;
                    const int64_t r = __ldcg(&lists[static_cast<uint64_t>(b) * a.listCap + (i - before)]);
                    const Vec16 tuple = ld_vec16(a.assist + r * 4);
                    uint2 ext = make_uint2(0u, 0u);
                    if (a.dedup != 0) ext = *reinterpret_cast<const uint2 *>(a.assistExt + r * 2);
                    CombineSendPart(a, comm, epoch, r, rows, static_cast<int>(tuple.x), static_cast<int64_t>(tuple.y) * KR + tuple.z, ext.x,
                                    ext.y, part, lane);
                }
            }
            PerfStageEnd(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC);
        } else if (sender) {
            PerfStageBegin(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC);
            // Unsorted: items are (chunk of rows, column part) in row order.
            const uint32_t c = a.chunkRows;
            const uint32_t nChunks = static_cast<uint32_t>((rows + c - 1) / c);
            const uint32_t nItems = nChunks * P;
            for (;;) {
                const uint32_t it = TakeItem(&cursors[0], lane);
                if (it >= nItems) break;
                const uint32_t chunk = it / P;
                const uint32_t part = it - chunk * P;
                const int64_t r = static_cast<int64_t>(chunk) * c + lane;
                int src = -1;
                int64_t slot = 0;
                uint2 ext = make_uint2(0u, 0u);
                uint32_t bucket = 0;
                const bool send = lane < static_cast<int>(c) && r < rows && classify(r, src, slot, ext, bucket);
                uint32_t m = __ballot_sync(0xffffffffu, send);
                while (m != 0) {
                    const int j = __ffs(m) - 1;
                    m &= m - 1;
                    const int64_t rj = static_cast<int64_t>(chunk) * c + j;
                    CombineSendPart(a, comm, epoch, rj, rows, __shfl_sync(0xffffffffu, src, j), __shfl_sync(0xffffffffu, slot, j),
                                    __shfl_sync(0xffffffffu, ext.x, j), __shfl_sync(0xffffffffu, ext.y, j), part, lane);
                }
            }
            PerfStageEnd(perf, TILEXR_PERF_LOCAL_INPUT_TO_IPC);
        }
        PerfStageBegin(perf, TILEXR_PERF_PEER_IPC_TO_OUTPUT);
        // ---- reduce this rank's tokens ------------------------------------------------------------------------
        const uint8_t *half = DataHalf(comm, rank, epoch);
        const uint32_t nReduce = static_cast<uint32_t>(a.bs) * P;
        while (w.ok()) {
            const uint32_t it = TakeItem(&cursors[1], lane);
            if (it >= nReduce) break;
            const int64_t t = it / P;
            const uint32_t part = it - static_cast<uint32_t>(t) * P;
            const int vBegin = static_cast<int>(part) * partVecs;
            const int vEnd = min(rowVecs, vBegin + partVecs);
            int e = -1;
            float wk = 0.f;
            unsigned long long myRowPtr = 0;
            const int64_t directRow = direct && lane < KR ? a.routeRows[t * KR + lane] : -1;     // beside the other loads, not behind them
            // `e` is the COLUMN of the route (shared ranks first, then routed experts), -1 when inactive
            if (lane < K) {
                e = a.expertIds != nullptr ? a.expertIds[t * K + lane] : 0;
                if (e >= a.numExperts) e = -1;
                if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_TOKEN && a.activeMask[t] == 0) e = -1;
                if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_EXPERT && a.activeMask[t * K + lane] == 0) e = -1;
                if (e >= 0) e += a.topo.sharedRanks;
                wk = a.expertScales != nullptr ? a.expertScales[t * K + lane] : 1.0f;
            } else if (lane < KR) {
                // the shared experts' outputs are added with weight one
                const bool activeTok = !(a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_TOKEN && a.activeMask[t] == 0);
                e = activeTok ? EpSharedCol(a.topo, rank, lane - K) : -1;
                wk = 1.0f;
            }
            const int myDst = e >= 0 ? EpColRank(a.topo, e) : -1;
            if (a.dedup != 0) {
                // routes to one remote rank come back as one weighted sum in the slot of the lowest k
                bool lower = false, higher = false;
                for (int j = 0; j < KR; ++j) {
                    const int dj = __shfl_sync(0xffffffffu, myDst, j);
                    if (dj >= 0 && dj == myDst && myDst != rank) {
                        if (j < lane) lower = true;
                        else if (j > lane) higher = true;
                    }
                }
                if (lower) e = -1;
                else if (higher) wk = 1.0f;
            }
            if (lane < KR && e >= 0) {
                const int64_t slot = t * KR + lane;
                const int64_t localRow = myDst == rank ? directRow : -1;
                if (localRow >= 0 && localRow < rows) {
                    myRowPtr = reinterpret_cast<unsigned long long>(a.expertOut + localRow * a.rowBytes);
                } else {
                    myRowPtr = reinterpret_cast<unsigned long long>(half + slot * a.rowBytes);
                    WaitFlagGE(w, FlagSlot(comm, rank, TILEXR_FLAG_SLOT_BASE + slot * P + part), 1, myDst, slot);
                }
            }
            const bool good = __all_sync(0xffffffffu, w.ok());
            if (!good) {
                if (w.ok()) w.status = TILEXR_DEV_ABORTED;
                break;
            }
            const uint32_t active = __ballot_sync(0xffffffffu, e >= 0);
            uint8_t *y = a.yOut + t * a.rowBytes;
            // RU 16-byte columns per lane and row: a warp reads RU * 512 contiguous bytes of a row in one go (DRAM
            // pages are used well although up to KR rows are walked together), and accumulates route by route
            // in k order.
            constexpr int RU = 2;
            for (int v0 = vBegin; v0 < vEnd; v0 += 32 * RU) {  // warp-uniform trip count: the loop body shuffles
                float acc[RU][8];
#pragma unroll
                for (int u = 0; u < RU; ++u) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[u][j] = 0.f;
                }
                for (int k = 0; k < KR; ++k) {
                    if (((active >> k) & 1u) == 0) continue;
                    const uint8_t *src = reinterpret_cast<const uint8_t *>(__shfl_sync(0xffffffffu, myRowPtr, k));
                    const float wgt = __shfl_sync(0xffffffffu, wk, k);
                    Vec16 q[RU];
#pragma unroll
                    for (int u = 0; u < RU; ++u) {
                        const int v = v0 + u * 32 + lane;
                        q[u] = Vec16{0u, 0u, 0u, 0u};
                        if (v < vEnd) q[u] = ld_vec16_stream(src + v * 16);
                    }
#pragma unroll
                    for (int u = 0; u < RU; ++u) {
                        float f[8];
                        Unpack8(q[u], bf16, f);
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[u][i] = fmaf(wgt, f[i], acc[u][i]);
                    }
                }
#pragma unroll
                for (int u = 0; u < RU; ++u) {
                    const int v = v0 + u * 32 + lane;
                    if (v >= vEnd) continue;
                    if (a.sharedExpertX != nullptr) {
                        float f[8];
                        Unpack8(ld_vec16(a.sharedExpertX + t * a.rowBytes + v * 16), bf16, f);
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[u][j] += f[j];
                    }
                    st_vec16(y + v * 16, Pack8(acc[u], bf16));
                }
            }
        }
        ok = w.ok();
        PerfStageEnd(perf, TILEXR_PERF_PEER_IPC_TO_OUTPUT);
    }
    ok = BlockBroadcastOk(ok);
    PerfStageEnd(perf, TILEXR_PERF_KERNEL_TOTAL);
    KernelEpilogue(w, ok, EP_SCRATCH_TOTALS_WORD);      // the cursors and the bucket counts
}

// Combine on one rank that knows the row of each of its routes: nothing is sent and nobody is waited for, so no block needs
// the others and the launch is an ordinary one.  A warp takes (token, column part) items, dealt out beforehand, and keeps the
// columns of up to eight routes' rows in flight; they are added in k order in fp32 and rounded once, as above.
// Bound by memory where the batch is large and by four dependent round trips (arguments, routes, rows, store) where it is small.
// EpCombineBody has its send part in the same registers and fetches two columns of one row at a time, a chain of sixteen round trips per
// warp for 16 tokens: 16 x 7168, top-8 13.5 us, 5.0 so; 1009 x 4096, top-6 14.7 and 13.2; 4096 x 7168 101 and 95.  Two or four columns
// of fewer rows at a time, or fewer warps with more, are slower (4096 x 7168 97 to 288 us, 1009 x 4096 15 to 57).
struct LocalRoute {
    float weight;
    int32_t row;       // -1: inactive, -2: active without a row
};

__device__ __forceinline__ LocalRoute LoadLocalRoute(const EpCombineArgs &a, int64_t t, int64_t rows, int lane)
{
    LocalRoute route{0.f, -1};
    if (lane < a.topK) {
        const int64_t i = t * a.topK + lane;
        const int e = a.expertIds[i];
        const int64_t row = a.routeRows[i];
        route.weight = a.expertScales != nullptr ? a.expertScales[i] : 1.0f;
        bool active = e >= 0 && e < a.numExperts;
        if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_TOKEN && a.activeMask[t] == 0) active = false;
        if (a.maskType == TileXREp::TILEXR_EP_ACTIVE_MASK_EXPERT && a.activeMask[i] == 0) active = false;
        if (active) route.row = row >= 0 && row < rows ? static_cast<int32_t>(row) : -2;
    }
    return route;
}

__device__ void EpCombineLocalBody(const EpCombineArgs &a)
{
    constexpr int KU = 8;              // routes whose columns are in flight together
    const int lane = threadIdx.x & 31;
    StreamRelease();
    StreamWait();
    Waiter w = MakeWaiter(a.comm, a.magic, blockIdx.x);
    PerfScope perf = PerfInit(threadIdx.x == 0 ? a.perfTrace : nullptr, static_cast<uint32_t>(a.comm->rank), blockIdx.x);
    PerfStageBegin(perf, TILEXR_PERF_KERNEL_TOTAL);
    PerfStageBegin(perf, TILEXR_PERF_PEER_IPC_TO_OUTPUT);
    const bool bf16 = a.isBf16 != 0;
    const int rowVecs = a.rowBytes / 16;
    const int64_t rows = a.sendCounts[a.sendCountEntries - 1];
    const int64_t items = static_cast<int64_t>(a.bs) * a.parts;
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (EP_LOCAL_THREADS / 32);
    int64_t it = static_cast<int64_t>(blockIdx.x) * (EP_LOCAL_THREADS / 32) + (threadIdx.x >> 5);
    LocalRoute next = it < items ? LoadLocalRoute(a, it / a.parts, rows, lane) : LocalRoute{0.f, -1};
    for (; it < items; it += warps) {
        const LocalRoute route = next;
        const int64_t t = it / a.parts;
        const int vBegin = static_cast<int>(it - t * a.parts) * static_cast<int>(a.partVecs);
        const int vEnd = min(rowVecs, vBegin + static_cast<int>(a.partVecs));
        const uint32_t active = __ballot_sync(0xffffffffu, route.row >= 0);
        if (__any_sync(0xffffffffu, route.row == -2)) {
            // the caller's ids name a route that the dispatch did not place (a world with peers waits for it and gives up)
            if (route.row == -2) RaiseFailure(w, TILEXR_DEV_WAIT_TIMEOUT, 0, t * a.topK + lane, static_cast<uint64_t>(rows), 0);
            break;
        }
        if (it + warps < items) next = LoadLocalRoute(a, (it + warps) / a.parts, rows, lane);     // on its way beside this item's rows
        uint8_t *y = a.yOut + t * a.rowBytes;
        for (int v0 = vBegin; v0 < vEnd; v0 += 32) {
            const int v = v0 + lane;
            float acc[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[j] = 0.f;
            for (int k0 = 0; k0 < a.topK; k0 += KU) {
                Vec16 q[KU];
#pragma unroll
                for (int u = 0; u < KU; ++u) {
                    const int32_t row = __shfl_sync(0xffffffffu, route.row, (k0 + u) & 31);
                    if (((active >> k0) >> u & 1u) != 0) {
                        const uint8_t *src = a.expertOut + static_cast<int64_t>(row) * a.rowBytes + static_cast<int64_t>(v) * 16;
                        if (v < vEnd) q[u] = ld_vec16_stream(src);
                    }
                }
#pragma unroll
                for (int u = 0; u < KU; ++u) {
                    const float wgt = __shfl_sync(0xffffffffu, route.weight, (k0 + u) & 31);
                    if (((active >> k0) >> u & 1u) != 0) {
                        float f[8];
                        Unpack8(q[u], bf16, f);
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[j] = fmaf(wgt, f[j], acc[j]);
                    }
                }
            }
            if (v >= vEnd) continue;
            if (a.sharedExpertX != nullptr) {
                float f[8];
                Unpack8(ld_vec16(a.sharedExpertX + t * a.rowBytes + static_cast<int64_t>(v) * 16), bf16, f);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] += f[j];
            }
            st_vec16(y + static_cast<int64_t>(v) * 16, Pack8(acc, bf16));
        }
    }
    PerfStageEnd(perf, TILEXR_PERF_PEER_IPC_TO_OUTPUT);
    PerfStageEnd(perf, TILEXR_PERF_KERNEL_TOTAL);
    // The launch counts like the others; one thread keeps the record without waiting for anybody.  Other blocks may still run: one that fails after this
    // overwrites the status, one that failed before is not overwritten.  (A block that only starts now would tag the abort word with the next
    // epoch; nothing but its being set is read.)  The last block to leave would know, but a counter that every block adds to behind its
    // stores takes 2.6 us of 1009 x 4096 tokens.
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        CommArgs *c = a.comm;
        c->dfx[TILEXR_DFX_MAGIC] = w.epoch;
        c->dfx[TILEXR_DFX_OP] = TILEXR_OP_EP_COMBINE;
        c->dfx[TILEXR_DFX_COUNT_ARG] = a.bs;
        auto *status = reinterpret_cast<unsigned long long *>(&c->dfx[TILEXR_DFX_RUN_STATUS]);
        atomicCAS(status, 0ull, static_cast<unsigned long long>(TILEXR_RUN_FINISHED));
        atomicCAS(status, static_cast<unsigned long long>(TILEXR_RUN_STARTED), static_cast<unsigned long long>(TILEXR_RUN_FINISHED));
        EndLocalLaunch(c, w);
    }
}

TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchKernel, EpDispatchArgs, EpDispatchBody<EP_PLAIN>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchKernelFp8, EpDispatchArgs, EpDispatchBody<EP_FP8>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchKernelMxfp8, EpDispatchArgs, EpDispatchBody<EP_MXFP8>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpDispatchKernelInt8, EpDispatchArgs, EpDispatchBody<EP_INT8>, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpCombineKernel, EpCombineArgs, EpCombineBody, EP_BLOCK_THREADS, 2)
TILEXR_DEFINE_KERNEL_OCC(TileXREpCombineLocalKernel, EpCombineArgs, EpCombineLocalBody, EP_LOCAL_THREADS, EP_LOCAL_BLOCKS_PER_SM)

// ---- stand-alone quantisation and norm kernels ---------------------------------------------------------------

// A thread per 16 elements, eight threads per 128-element block.  h is a multiple of 128, so a block's threads are
// neighbours in one warp and rows need no alignment to warps: a short batch of long rows still fills the chip (a warp per
// row walking along it took 8.7 us for 2048 x 4096, this takes 5.9).
// `f` holds this thread's elements; writes its 16 fp8 values and, from the first thread of a block, the block's scale.
__device__ __forceinline__ void Fp8QuantStore16(const float *f, int64_t idx, uint32_t blockMask, uint8_t *y, float *scales)
{
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
    amax = fmaxf(amax, __shfl_xor_sync(blockMask, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(blockMask, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(blockMask, amax, 4));
    amax = fmaxf(amax, FP8_AMAX_FLOOR);
    const float inv = FP8_E4M3_MAX / amax;
    if ((idx & 7) == 0) scales[idx >> 3] = amax / FP8_E4M3_MAX;
    Vec16 q;
    q.x = Fp8x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
    q.y = Fp8x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
    q.z = Fp8x4(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
    q.w = Fp8x4(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
    st_vec16(y + idx * 16, q);
}

__global__ void __launch_bounds__(256) Fp8Quant1x128Kernel(const uint8_t *x, int64_t vecs, int bf16, uint8_t *y, float *scales)
{
    StreamRelease();
    StreamWait();
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= vecs) return;          // vecs is a multiple of eight: the threads of a 128-element block leave together
    float f[16];
    Unpack8(ld_vec16(x + idx * 32), bf16 != 0, f);
    Unpack8(ld_vec16(x + idx * 32 + 16), bf16 != 0, f + 8);
    Fp8QuantStore16(f, idx, 0xffu << (threadIdx.x & 24), y, scales);
}

// silu(gate) * up of rows [gate (f elements) | up (f elements)], computed in fp32 and rounded to the 16-bit type; with
// `scales` the rounded values are then quantised as above, else they are stored.  One pass instead of the four to six
// elementwise launches (and their fp32 copies of both halves) of the unfused form: 146 + 11 -> 21 us for 2048 rows of 2 x 7168.
// Bound by the arithmetic (an exponential and a division per output; the SMs 79 % busy, DRAM 46 % at 8192 rows).  A kernel per 16-bit type: with the
// type read at run time the conversions of both are in the way (8192 rows of 2 x 7168: 69.3 us with fp8 output and 69.2 without, 66.4 and 67.5 so).
template <bool BF16>
__device__ __forceinline__ void Swiglu8(const uint8_t *gate, const uint8_t *up, float *o)
{
    float g[8], u[8];
    Unpack8(ld_vec16(gate), BF16, g);
    Unpack8(ld_vec16(up), BF16, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = g[j] / (1.0f + expf(-g[j])) * u[j];
}

template <bool BF16>
__global__ void __launch_bounds__(256) SwigluKernel(const uint8_t *gateUp, int64_t vecs, int vecsPerRow, uint8_t *y)
{
    StreamRelease();
    StreamWait();
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;     // a thread per 8 outputs
    if (idx >= vecs) return;
    const int64_t row = idx / vecsPerRow;
    const uint8_t *gate = gateUp + (idx + row * vecsPerRow) * 16;                         // row r starts at vector 2 r vecsPerRow
    float o[8];
    Swiglu8<BF16>(gate, gate + static_cast<int64_t>(vecsPerRow) * 16, o);
    st_vec16(y + idx * 16, Pack8(o, BF16));
}

template <bool BF16>
__global__ void __launch_bounds__(256) SwigluFp8Quant1x128Kernel(const uint8_t *gateUp, int64_t vecs, int vecsPerRow, uint8_t *y, float *scales)
{
    StreamRelease();
    StreamWait();
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;     // a thread per 16 outputs
    if (idx >= vecs) return;
    const int64_t row = idx / vecsPerRow;
    const uint8_t *gate = gateUp + (idx + row * vecsPerRow) * 32;
    const uint8_t *up = gate + static_cast<int64_t>(vecsPerRow) * 32;
    float f[16];
    Swiglu8<BF16>(gate, up, f);
    Swiglu8<BF16>(gate + 16, up + 16, f + 8);
    Unpack8(Pack8(f, BF16), BF16, f);              // quantise what the unfused form stores
    Unpack8(Pack8(f + 8, BF16), BF16, f + 8);
    Fp8QuantStore16(f, idx, 0xffu << (threadIdx.x & 24), y, scales);
}

// Eight fp8 values times a scale.
constexpr int DEQUANT_STEPS = 4;

// Bound by memory: 32768 x 7168 reads 242 MB and writes 470 MB, 142 us with one step, a 64-bit division and a row index per thread, 107 us so (6.7 TB/s).
__global__ void __launch_bounds__(256) Fp8Dequant1x128Kernel(const uint8_t *y, const float *scales, int64_t vecs, int bf16, uint8_t *x)
{
    StreamRelease();
    StreamWait();
    // Eight elements per thread and step, DEQUANT_STEPS steps with all their loads first.  h is a multiple of 128, so the
    // matrix is one run of vectors and vector i has scale i / 16: no division by the row length.
    const int64_t base = static_cast<int64_t>(blockIdx.x) * (blockDim.x * DEQUANT_STEPS) + threadIdx.x;
    uint2 raw[DEQUANT_STEPS];
    float s[DEQUANT_STEPS];
#pragma unroll
    for (int u = 0; u < DEQUANT_STEPS; ++u) {
        const int64_t i = base + u * static_cast<int64_t>(blockDim.x);
        if (i < vecs) {
            raw[u] = __ldcs(reinterpret_cast<const uint2 *>(y) + i);
            s[u] = scales[i >> 4];
        }
    }
#pragma unroll
    for (int u = 0; u < DEQUANT_STEPS; ++u) {
        const int64_t i = base + u * static_cast<int64_t>(blockDim.x);
        if (i >= vecs) break;
        float f[8];
        Fp8Unpack8(raw[u], __NV_E4M3, s[u], f);
        st_vec16(x + i * 16, Pack8(f, bf16 != 0));
    }
}

// MXFP8: 32-element blocks share an E8M0 exponent 2^(floor(log2(amax)) - emax), emax = 8 for
// e4m3 and 15 for e5m2; elements are x / 2^exp rounded to nearest even with saturation.
__global__ void __launch_bounds__(256) Mxfp8QuantKernel(const uint8_t *x, int64_t rows, int h, int bf16, int e5m2, uint8_t *y, uint8_t *scales)
{
    const int blocksPerRow = (h + 31) / 32;
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;   // one thread per 32-element block
    if (idx >= rows * blocksPerRow) return;
    const int64_t row = idx / blocksPerRow;
    const int b = static_cast<int>(idx % blocksPerRow);
    const int n = min(32, h - b * 32);
    float f[32];
    float amax = 0.f;
    for (int j = 0; j < 32; ++j) {
        float v = 0.f;
        if (j < n) {
            const uint16_t raw = *reinterpret_cast<const uint16_t *>(x + (row * h + b * 32 + j) * 2);
            v = bf16 ? __uint_as_float(static_cast<uint32_t>(raw) << 16) : __half2float(*reinterpret_cast<const __half *>(&raw));
        }
        f[j] = v;
        amax = fmaxf(amax, fabsf(v));
    }
    const int emax = e5m2 ? 15 : 8;
    int exp = 0;
    if (amax > 0.f) {
        exp = static_cast<int>((__float_as_uint(amax) >> 23) & 0xff) - 127 - emax;   // floor(log2(amax)) - emax
        if ((__float_as_uint(amax) >> 23) == 0) exp = -126 - emax;                    // subnormal input
    } else {
        exp = -127;
    }
    exp = max(-127, min(127, exp));
    scales[row * blocksPerRow + b] = static_cast<uint8_t>(exp + 127);
    const float inv = exp2f(static_cast<float>(-exp));
    for (int j = 0; j < n; ++j) {
        const float v = f[j] * inv;
        const __nv_fp8_storage_t q = __nv_cvt_float_to_fp8(v, __NV_SATFINITE, e5m2 ? __NV_E5M2 : __NV_E4M3);
        y[row * h + b * 32 + j] = q;
    }
}

__global__ void __launch_bounds__(256) Mxfp8DequantKernel(const uint8_t *y, const uint8_t *scales, int64_t rows, int h, int e5m2, int bf16, uint8_t *x)
{
    const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= rows * h) return;
    const int64_t row = idx / h;
    const int col = static_cast<int>(idx % h);
    const int blocksPerRow = (h + 31) / 32;
    const float s = exp2f(static_cast<float>(static_cast<int>(scales[row * blocksPerRow + col / 32]) - 127));
    const __half_raw hr = __nv_cvt_fp8_to_halfraw(y[idx], e5m2 ? __NV_E5M2 : __NV_E4M3);
    const float v = __half2float(*reinterpret_cast<const __half *>(&hr)) * s;
    if (bf16) {
        const __nv_bfloat16 o = __float2bfloat16_rn(v);
        *reinterpret_cast<__nv_bfloat16 *>(x + idx * 2) = o;
    } else {
        *reinterpret_cast<__half *>(x + idx * 2) = __float2half_rn(v);
    }
}

// MXFP8 rows whose length is a multiple of eight (a group of eight elements then lies in one 32-element block and its 16
// bytes of output are aligned): eight elements per thread instead of one.  32768 x 7168: 783 -> 139 us, 132 with a
// kernel per pair of types and without a division per vector where rows are whole blocks.
template <bool E5M2, bool BF16>
__global__ void __launch_bounds__(256) Mxfp8Dequant8Kernel(const uint8_t *y, const uint8_t *scales, int64_t vecs, int vecsPerRow, int blocksPerRow, uint8_t *x)
{
    StreamRelease();
    StreamWait();
    const int64_t base = static_cast<int64_t>(blockIdx.x) * (blockDim.x * DEQUANT_STEPS) + threadIdx.x;
    uint2 raw[DEQUANT_STEPS];
    int exponent[DEQUANT_STEPS];
#pragma unroll
    for (int u = 0; u < DEQUANT_STEPS; ++u) {
        const int64_t i = base + u * static_cast<int64_t>(blockDim.x);
        if (i < vecs) {
            raw[u] = __ldcs(reinterpret_cast<const uint2 *>(y) + i);
            int64_t at = i >> 2;                                       // rows of whole 32-element blocks: vector i has scale i / 4
            if (vecsPerRow != 4 * blocksPerRow) {
                const int64_t row = i / vecsPerRow;
                at = row * blocksPerRow + (i - row * vecsPerRow) / 4;
            }
            exponent[u] = static_cast<int>(scales[at]) - 127;
        }
    }
#pragma unroll
    for (int u = 0; u < DEQUANT_STEPS; ++u) {
        const int64_t i = base + u * static_cast<int64_t>(blockDim.x);
        if (i >= vecs) break;
        float f[8];
        Fp8Unpack8(raw[u], E5M2 ? __NV_E5M2 : __NV_E4M3, exp2f(static_cast<float>(exponent[u])), f);
        st_vec16(x + i * 16, Pack8(f, BF16));
    }
}

// Gradients of a weighted combine with respect to the expert rows and the gate weights, a warp per row r of the dispatched
// output gradient g:   gradRows[r] = w[r] * g[r] (fp32, rounded once)   and   dot[r] = <g[r], rows[r]> (fp32).
// The dot product goes to columns 2 slot and 2 slot + 1 of wide[r] as a (high, low) bf16 pair and zeros to the other columns,
// the row that a narrow combine then returns to its token.  Rows past *rowCount are nobody's: their gradient is zero.
// `rows` is null where the gate weights need no gradient.  One pass over g and rows, bound by memory, instead of the fp32
// copies, products and reductions of the unfused form: 16384 x 4096, about 970 us in nine launches, 62 us so (6.6 TB/s).
__global__ void __launch_bounds__(256) CombineBackwardKernel(const uint8_t *g, const float *weights, const uint8_t *rows, const int32_t *assist,
                                                             const int32_t *rowCount, int64_t capacity, int vecsPerRow, int bf16, int slots,
                                                             int wideVecs, uint8_t *gradRows, uint8_t *wide)
{
    const int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (r >= capacity) return;
    const bool used = r < *rowCount;
    const uint8_t *gRow = g + r * vecsPerRow * 16;
    const uint8_t *outRow = rows + r * vecsPerRow * 16;
    uint8_t *gradRow = gradRows + r * vecsPerRow * 16;
    if (!used) {
        for (int v = lane; v < vecsPerRow; v += 32) st_vec16(gradRow + v * 16, Vec16{0u, 0u, 0u, 0u});
        return;
    }
    const float w = weights[r];
    float dot = 0.f;
    constexpr int U = 4;
    for (int v0 = lane; v0 < vecsPerRow; v0 += 32 * U) {
        Vec16 a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32;
            if (v < vecsPerRow) {
                a[u] = ld_vec16_stream(gRow + v * 16);
                if (rows != nullptr) b[u] = ld_vec16_stream(outRow + v * 16);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32;
            if (v >= vecsPerRow) break;
            float f[8], o[8];
            Unpack8(a[u], bf16 != 0, f);
            if (rows != nullptr) {
                Unpack8(b[u], bf16 != 0, o);
#pragma unroll
                for (int j = 0; j < 8; ++j) dot = fmaf(f[j], o[j], dot);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] *= w;
            st_vec16(gradRow + v * 16, Pack8(f, bf16 != 0));
        }
    }
    if (rows == nullptr) return;
    dot = WarpSum(dot);
    const __nv_bfloat16 high = __float2bfloat16_rn(dot);
    const __nv_bfloat162 pair = __halves2bfloat162(high, __float2bfloat16_rn(dot - __bfloat162float(high)));
    const int slot = max(0, min(slots - 1, assist[r * 4 + 2]));
    for (int v = lane; v < wideVecs; v += 32) {
        uint32_t q[4] = {0u, 0u, 0u, 0u};
        if (slot >> 2 == v) q[slot & 3] = *reinterpret_cast<const uint32_t *>(&pair);
        st_vec16(wide + (r * wideVecs + v) * 16, Vec16{q[0], q[1], q[2], q[3]});
    }
}

// The same on one rank, from the output gradient where it is: the row of every route is known from the forward dispatch, so grad_y
// needs no dispatch of its own (which wrote topK copies of it for this kernel to read) and the dot products no way back.  A warp
// per route; the topK warps of a token are neighbours and find its gradient in L2.  Bound by reading the expert rows and writing
// their gradients: 2048 x 4096, top-8 48 us (5.9 TB/s), where the dispatch, the kernel above and the narrow combine took 130.
__global__ void __launch_bounds__(256) CombineBackwardLocalKernel(const uint8_t *gradY, const float *weights, const uint8_t *rows, const int32_t *routeRows,
                                                                  const int32_t *rowCount, int64_t routes, int topK, int64_t capacity, int vecsPerRow,
                                                                  int bf16, uint8_t *gradRows, float *gradWeights)
{
    StreamRelease();
    StreamWait();
    const int64_t i = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (i >= *rowCount && i < capacity) {           // a row that no route fills
        for (int v = lane; v < vecsPerRow; v += 32) st_vec16(gradRows + (i * vecsPerRow + v) * 16, Vec16{0u, 0u, 0u, 0u});
    }
    if (i >= routes) return;
    const int64_t r = routeRows[i];
    if (r < 0 || r >= capacity) {
        if (gradWeights != nullptr && lane == 0) gradWeights[i] = 0.f;
        return;
    }
    const float w = weights[i];
    const uint8_t *gRow = gradY + (i / topK) * vecsPerRow * 16;
    const uint8_t *outRow = rows + r * vecsPerRow * 16;
    uint8_t *gradRow = gradRows + r * vecsPerRow * 16;
    float dot = 0.f;
    constexpr int U = 4;
    for (int v0 = lane; v0 < vecsPerRow; v0 += 32 * U) {
        Vec16 a[U], b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32;
            if (v < vecsPerRow) {
                a[u] = ld_vec16(gRow + v * 16);
                if (gradWeights != nullptr) b[u] = ld_vec16_stream(outRow + v * 16);
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int v = v0 + u * 32;
            if (v >= vecsPerRow) break;
            float f[8], o[8];
            Unpack8(a[u], bf16 != 0, f);
            if (gradWeights != nullptr) {
                Unpack8(b[u], bf16 != 0, o);
#pragma unroll
                for (int j = 0; j < 8; ++j) dot = fmaf(f[j], o[j], dot);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] *= w;
            st_vec16(gradRow + v * 16, Pack8(f, bf16 != 0));
        }
    }
    if (gradWeights == nullptr) return;
    dot = WarpSum(dot);
    if (lane == 0) gradWeights[i] = dot;
}

// One block per row.  The row stays in registers between the two passes.
__global__ void __launch_bounds__(256) RmsNormKernel(const uint8_t *x, uint8_t *residual, const uint8_t *gamma, float eps, int h, int bf16, uint8_t *y)
{
    __shared__ float partial[8];
    const int64_t row = blockIdx.x;
    const int vecs = h / 8;
    constexpr int MAX_VECS = 8;   // 256 threads x 8 vectors x 8 elements = 16384 columns
    float vals[MAX_VECS][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < MAX_VECS; ++i) {
        const int v = i * 256 + threadIdx.x;
        if (v < vecs) {
            Unpack8(ld_vec16(x + (row * h + static_cast<int64_t>(v) * 8) * 2), bf16 != 0, vals[i]);
            if (residual != nullptr) {
                float r[8];
                Unpack8(ld_vec16(residual + (row * h + static_cast<int64_t>(v) * 8) * 2), bf16 != 0, r);
#pragma unroll
                for (int j = 0; j < 8; ++j) vals[i][j] += r[j];
                // the sum, rounded to the storage type, is both the new residual and the norm input
                const Vec16 packed = Pack8(vals[i], bf16 != 0);
                st_vec16(residual + (row * h + static_cast<int64_t>(v) * 8) * 2, packed);
                Unpack8(packed, bf16 != 0, vals[i]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) ss += vals[i][j] * vals[i][j];
        }
    }
    ss = WarpSum(ss);
    if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) tot += partial[i];
    const float rstd = rsqrtf(tot / static_cast<float>(h) + eps);
#pragma unroll
    for (int i = 0; i < MAX_VECS; ++i) {
        const int v = i * 256 + threadIdx.x;
        if (v < vecs) {
            float g[8];
            Unpack8(ld_vec16(gamma + static_cast<int64_t>(v) * 16), bf16 != 0, g);
            float o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = vals[i][j] * rstd * g[j];
            st_vec16(y + (row * h + static_cast<int64_t>(v) * 8) * 2, Pack8(o, bf16 != 0));
        }
    }
}

// A launch of 256-thread blocks of a kernel that calls StreamWait; CheckLaunch finds its error.
template <typename... P, typename... A> void LaunchSimple(void (*kernel)(P...), unsigned grid, void *stream, A... args)
{
    std::tuple<P...> values(static_cast<P>(args)...);
    std::apply(
        [&](auto &...v) {
            void *params[] = {const_cast<void *>(static_cast<const void *>(&v))...};
            LaunchOverlapped(reinterpret_cast<const void *>(kernel), grid, 1, 256, 0, 0, params, stream);
        },
        values);
}

int CheckLaunch(const char *what)
{
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        fprintf(stderr, "[TileXR] %s launch failed: %s\n", what, cudaGetErrorString(e));
        return TILEXR_ERROR_RUNTIME;
    }
    NoteLaunch();
    return TILEXR_SUCCESS;
}

} // namespace

const KernelEntry &EpDispatchKernelEntry(int64_t quantMode)
{
    switch (quantMode) {
        case TileXREp::TILEXR_EP_QUANT_FP8_1X128: return TileXREpDispatchKernelFp8Entry;
        case TileXREp::TILEXR_EP_QUANT_MXFP8_E4M3:
        case TileXREp::TILEXR_EP_QUANT_MXFP8_E5M2: return TileXREpDispatchKernelMxfp8Entry;
        case TileXREp::TILEXR_EP_QUANT_STATIC_INT8:
        case TileXREp::TILEXR_EP_QUANT_DYNAMIC_INT8: return TileXREpDispatchKernelInt8Entry;
        default: return TileXREpDispatchKernelEntry;
    }
}
const KernelEntry &EpCombineLocalKernelEntry() { return TileXREpCombineLocalKernelEntry; }
const KernelEntry &EpCombineKernelEntry() { return TileXREpCombineKernelEntry; }

size_t EpDispatchSmemBytes(int numExperts, int routesPerBlock)
{
    return static_cast<size_t>(routesPerBlock) * 8 + static_cast<size_t>(numExperts) * 20 + 4 + EP_WARPS * 64 * sizeof(float);
}

int LaunchRoutingTopK(const RoutingArgs &args, void *stream)
{
    const int warpsPerBlock = 8;
    const unsigned grid = static_cast<unsigned>((args.bs + warpsPerBlock - 1) / warpsPerBlock);
    RoutingTopKKernel<<<grid, warpsPerBlock * 32, 0, static_cast<cudaStream_t>(stream)>>>(args);
    return CheckLaunch("routing top-k");
}

int LaunchFp8Quant1x128(const void *x, int64_t rows, int64_t h, bool bf16, void *y, float *scales, void *stream)
{
    const int64_t vecs = rows * (h / 16);
    LaunchSimple(Fp8Quant1x128Kernel, static_cast<unsigned>((vecs + 255) / 256), stream,
                 static_cast<const uint8_t *>(x), vecs, bf16 ? 1 : 0, static_cast<uint8_t *>(y), scales);
    return CheckLaunch("fp8 quant");
}

int LaunchSwiglu(const void *gateUp, int64_t rows, int64_t f, bool bf16, void *y, float *scales, void *stream)
{
    if (scales != nullptr) {
        const int64_t vecs = rows * (f / 16);
        LaunchSimple(bf16 ? SwigluFp8Quant1x128Kernel<true> : SwigluFp8Quant1x128Kernel<false>, static_cast<unsigned>((vecs + 255) / 256), stream,
                     static_cast<const uint8_t *>(gateUp), vecs, static_cast<int>(f / 16), static_cast<uint8_t *>(y), scales);
        return CheckLaunch("swiglu fp8 quant");
    }
    const int64_t vecs = rows * (f / 8);
    LaunchSimple(bf16 ? SwigluKernel<true> : SwigluKernel<false>, static_cast<unsigned>((vecs + 255) / 256), stream,
                 static_cast<const uint8_t *>(gateUp), vecs, static_cast<int>(f / 8), static_cast<uint8_t *>(y));
    return CheckLaunch("swiglu");
}

int LaunchFp8Dequant1x128(const void *y, const float *scales, int64_t rows, int64_t h, bool bf16, void *x, void *stream)
{
    const int64_t n = rows * (h / 8);
    const unsigned grid = static_cast<unsigned>((n + 256 * DEQUANT_STEPS - 1) / (256 * DEQUANT_STEPS));
    LaunchSimple(Fp8Dequant1x128Kernel, grid, stream, static_cast<const uint8_t *>(y), scales, n, bf16 ? 1 : 0, static_cast<uint8_t *>(x));
    return CheckLaunch("fp8 dequant");
}

int LaunchMxfp8Quant(const void *x, int64_t rows, int64_t h, bool bf16, bool e5m2, void *y, uint8_t *scales, void *stream)
{
    const int64_t n = rows * ((h + 31) / 32);
    const unsigned grid = static_cast<unsigned>((n + 255) / 256);
    Mxfp8QuantKernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint8_t *>(x), rows, static_cast<int>(h),
                                                                           bf16 ? 1 : 0, e5m2 ? 1 : 0, static_cast<uint8_t *>(y), scales);
    return CheckLaunch("mxfp8 quant");
}

int LaunchMxfp8Dequant(const void *y, const uint8_t *scales, int64_t rows, int64_t h, bool e5m2, bool bf16, void *x, void *stream)
{
    if (h % 8 == 0 && ((reinterpret_cast<uintptr_t>(y) & 7u) | (reinterpret_cast<uintptr_t>(x) & 15u)) == 0) {
        const int64_t vecs = rows * (h / 8);
        const auto kernel = e5m2 ? (bf16 ? Mxfp8Dequant8Kernel<true, true> : Mxfp8Dequant8Kernel<true, false>)
                                 : (bf16 ? Mxfp8Dequant8Kernel<false, true> : Mxfp8Dequant8Kernel<false, false>);
        LaunchSimple(kernel, static_cast<unsigned>((vecs + 256 * DEQUANT_STEPS - 1) / (256 * DEQUANT_STEPS)), stream,
                     static_cast<const uint8_t *>(y), scales, vecs, static_cast<int>(h / 8), static_cast<int>((h + 31) / 32), static_cast<uint8_t *>(x));
        return CheckLaunch("mxfp8 dequant");
    }
    const int64_t n = rows * h;
    const unsigned grid = static_cast<unsigned>((n + 255) / 256);
    Mxfp8DequantKernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const uint8_t *>(y), scales, rows,
                                                                             static_cast<int>(h), e5m2 ? 1 : 0, bf16 ? 1 : 0,
                                                                             static_cast<uint8_t *>(x));
    return CheckLaunch("mxfp8 dequant");
}

int LaunchCombineBackward(const void *g, const float *weights, const void *rows, const int32_t *assist, const int32_t *rowCount, int64_t capacity,
                          int64_t h, bool bf16, int slots, int wideCols, void *gradRows, void *wide, void *stream)
{
    CombineBackwardKernel<<<static_cast<unsigned>((capacity + 7) / 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t *>(g), weights, static_cast<const uint8_t *>(rows), assist, rowCount, capacity, static_cast<int>(h / 8), bf16 ? 1 : 0,
        slots, wideCols / 8, static_cast<uint8_t *>(gradRows), static_cast<uint8_t *>(wide));
    return CheckLaunch("combine backward");
}

int LaunchCombineBackwardLocal(const void *gradY, const float *weights, const void *rows, const int32_t *routeRows, const int32_t *rowCount, int64_t bs,
                               int64_t topK, int64_t capacity, int64_t h, bool bf16, void *gradRows, float *gradWeights, void *stream)
{
    const int64_t warps = std::max(bs * topK, capacity);
    LaunchSimple(CombineBackwardLocalKernel, static_cast<unsigned>((warps + 7) / 8), stream,
                 static_cast<const uint8_t *>(gradY), weights, static_cast<const uint8_t *>(rows), routeRows, rowCount, bs * topK, static_cast<int>(topK), capacity, static_cast<int>(h / 8), bf16 ? 1 : 0, static_cast<uint8_t *>(gradRows), gradWeights);
    return CheckLaunch("combine backward on one rank");
}

int LaunchRmsNorm(const void *x, void *residual, const void *gamma, float eps, int64_t rows, int64_t h, bool bf16, void *y, void *stream)
{
    RmsNormKernel<<<static_cast<unsigned>(rows), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const uint8_t *>(x), static_cast<uint8_t *>(residual), static_cast<const uint8_t *>(gamma), eps,
        static_cast<int>(h), bf16 ? 1 : 0, static_cast<uint8_t *>(y));
    return CheckLaunch("rmsnorm");
}

} // namespace TileXR
