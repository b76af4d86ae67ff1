// bf16/fp16 GEMM for few rows: the weight is the tall operand of the tensor cores.
//
//   C[M,N] = A[M,K] x B[N,K]^T, computed as tiles of C^T: 128 rows of B (output columns) x `tn` rows of A (16 to 128)
//
// A product of a handful of rows is bound by reading the weight once.  The 256 x 256 tiles of the CTA-pair kernel then fill
// most of the tensor cores' work and of the shared-memory ring with rows that do not exist, and N / 256 tiles leave most SMs
// without any: 17 x 7168 x 2048 ran on 28 SMs.  Here a tile takes 16 KB of weight and 2 to 16 KB of rows per 64-wide
// step of K, two CTAs share an SM (about 180 KB of loads in flight per SM), and where there are fewer tiles than places
// the CTAs of a cluster split K: each keeps its partial tile in tensor memory, sends every other CTA a slice of columns
// through distributed shared memory and adds the slices it receives in split order, so the result does not depend on timing.
//
// The grouped form (row counts per group on the device, as in the CTA-pair kernel) walks (group, chunk of tn rows) x weight
// tiles with persistent CTAs; chunks of one group are neighbours, so a second chunk finds the weight in L2.
//
// Roles per CTA (192 threads): warp 0 TMA, warp 1 tensor memory and MMA, warps 2-5 epilogue.  Every mbarrier wait is bounded;
// on a give-up all roles fall through to the cluster barriers and the tear-down, no CTA of the cluster stores a sum that the part is
// missing from, and `status`, where the caller gives one, tells the host.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "device/tilexr_rma.cuh"
#include "gemm_kernels.cuh"
#include "tilexr_types.h"

namespace TileXR {

using namespace tilexr;

namespace {

struct SkinnyState {
    uint64_t full[GEMM_SKINNY_MAX_STAGES];
    uint64_t empty[GEMM_SKINNY_MAX_STAGES];
    uint64_t tmemFull[2];
    uint64_t tmemEmpty[2];
    uint32_t tmemBase;
    volatile int abortFlag;
};
static_assert(sizeof(SkinnyState) <= GEMM_SKINNY_STATE_BYTES, "barriers fit their slot");

__device__ __forceinline__ void SkTmaLoad(void *smemDst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(SmemAddr(smemDst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(SmemAddr(bar))
        : "memory");
}

__device__ __forceinline__ void SkFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void SkFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void SkClusterSync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// K-major tile written by TMA with 128-byte swizzle: rows 128 bytes apart, groups of eight rows 1024 bytes apart.
__device__ __forceinline__ uint64_t SkSmemDesc(uint32_t smemAddr)
{
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smemAddr & 0x3ffffu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

__device__ __forceinline__ void SkUmma(uint32_t tmemD, uint64_t descA, uint64_t descB, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n"
        ::"r"(tmemD), "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void SkCommit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(SmemAddr(bar)) : "memory");
}

// Sixteen columns of this warp's 32 lanes, complete when the statement is done.
__device__ __forceinline__ void SkTmemLoad16(uint32_t taddr, uint32_t *r)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// Bounded wait of a whole warp with one verdict for all lanes.
__device__ __forceinline__ bool SkWait(uint64_t *bar, uint32_t parity, SkinnyState *st)
{
    bool done = MbarTryWait(bar, parity);
    if (!done) {
        uint64_t deadline = 0;
        for (uint32_t polls = 1;; ++polls) {
            done = MbarTryWait(bar, parity);
            if (done) break;
            if ((polls & 127u) == 0) {
                if (st->abortFlag != 0) break;
                const uint64_t t = now_ns();
                if (deadline == 0) {
                    deadline = t + 4000000000ull;
                } else if (t > deadline) {
                    st->abortFlag = 1;
                    break;
                }
            }
        }
    }
    return __all_sync(0xffffffffu, done) != 0;
}

struct SkinnyTile {
    int row0, rowEnd;      // rows of A and C
    int n0;                // first output column
    int rowW;              // first row of B
};

__device__ __forceinline__ SkinnyTile SkTileOf(const SkinnyArgs &a, int item, const int *rowStart, const int *chunkStart, int mTiles)
{
    SkinnyTile t;
    if (a.groupRows == nullptr) {
        const int wTile = item / mTiles;                       // the row tiles of one weight tile are neighbours
        t.row0 = (item - wTile * mTiles) * a.tn;
        t.rowEnd = a.M;
        t.n0 = wTile * 128;
        t.rowW = t.n0;
        return t;
    }
    const int chunk = item / a.nTiles;
    int lo = 0, hi = a.groups - 1;                             // last group whose first chunk is at or before `chunk`
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (chunkStart[mid] <= chunk) lo = mid;
        else hi = mid - 1;
    }
    t.row0 = rowStart[lo] + (chunk - chunkStart[lo]) * a.tn;
    t.rowEnd = rowStart[lo + 1];
    t.n0 = (item - chunk * a.nTiles) * 128;
    t.rowW = (a.groupBase + lo) * a.N + t.n0;
    return t;
}

// One output value per lane (lane = output column n, the same row of C for the whole warp).
__device__ __forceinline__ void SkStore(const SkinnyArgs &a, float v, int n, int row, int lane)
{
    const bool bf16 = a.isBf16 != 0;
    float o = v;
    int col = n, cols = a.N;
    bool mine = n < a.N;
    if (a.epilogue == GEMM_EPI_SWIGLU) {
        const float up = __shfl_xor_sync(0xffffffffu, v, 1);   // weight row 2i gate, 2i + 1 up: neighbouring lanes
        o = v / (1.0f + __expf(-v)) * up;
        col = n >> 1;
        cols = a.N >> 1;
        mine = mine && (lane & 1) == 0;
    }
    if (mine) {
        uint8_t *p = a.c + (static_cast<uint64_t>(row) * cols + col) * 2;
        if (bf16) *reinterpret_cast<__nv_bfloat16 *>(p) = __float2bfloat16_rn(o);
        else *reinterpret_cast<__half *>(p) = __float2half_rn(o);
    }
}

__global__ void __launch_bounds__(GEMM_SKINNY_THREADS, 2) TileXRGemmSkinny(const __grid_constant__ SkinnyArgs a)
{
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    const uint32_t stageBytes = GEMM_SKINNY_W_BYTES + static_cast<uint32_t>(a.tn) * 128u;
    SkinnyState *st = reinterpret_cast<SkinnyState *>(smem + a.stages * stageBytes);
    int *rowStart = reinterpret_cast<int *>(smem + a.stages * stageBytes + GEMM_SKINNY_STATE_BYTES);
    int *chunkStart = rowStart + GEMM_SKINNY_MAX_GROUPS + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int split = a.split;
    const int part = static_cast<int>(blockIdx.x) % split;     // clusters are `split` consecutive CTAs
    uint32_t tmemCols = 32;
    while (tmemCols < 2u * a.tn) tmemCols *= 2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            MbarInit(&st->full[s], 1);
            MbarInit(&st->empty[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            MbarInit(&st->tmemFull[i], 1);
            MbarInit(&st->tmemEmpty[i], 4);
        }
        st->abortFlag = 0;
        MbarInitFence();
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&a.tmapW)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&a.tmapX)) : "memory");
    }
    StreamRelease();
    StreamWait();
    if (a.groupRows != nullptr && warp == 2) BuildGroupTable(a.groupRows, a.groupBase, a.groups, a.M, a.tn, lane, rowStart, chunkStart);
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(&st->tmemBase)), "r"(tmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    SkFenceBefore();
    __syncthreads();
    SkFenceAfter();
    const uint32_t tmemBase = st->tmemBase;

    const int mTiles = (a.M + a.tn - 1) / a.tn;
    const int items = (a.groupRows != nullptr ? chunkStart[a.groups] : mTiles) * a.nTiles;
    const int first = static_cast<int>(blockIdx.x) / split;
    const int step = static_cast<int>(gridDim.x) / split;
    const int kPer = (a.kBlocks + split - 1) / split;
    const int k0 = part * kPer;
    const int k1 = min(a.kBlocks, k0 + kPer);

    if (warp == 0) {
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (int item = first; item < items && ok; item += step) {
            const SkinnyTile t = SkTileOf(a, item, rowStart, chunkStart, mTiles);
            for (int kb = k0; kb < k1; ++kb) {
                ok = SkWait(&st->empty[stage], phase ^ 1u, st);
                if (!ok) break;
                if (ElectOne()) {
                    uint8_t *sw = smem + stage * stageBytes;
                    MbarExpectTx(&st->full[stage], stageBytes);
                    SkTmaLoad(sw, &a.tmapW, kb * GEMM_BK, t.rowW, &st->full[stage]);
                    SkTmaLoad(sw + GEMM_SKINNY_W_BYTES, &a.tmapX, kb * GEMM_BK, t.row0, &st->full[stage]);
                }
                if (++stage == static_cast<uint32_t>(a.stages)) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        const uint32_t fmt = a.isBf16 != 0 ? 1u : 0u;
        const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(a.tn >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
        const uint64_t desc0 = SkSmemDesc(SmemAddr(smem));
        uint32_t stage = 0, phase = 0;
        int iter = 0;
        bool ok = true;
        for (int item = first; item < items && ok; item += step, ++iter) {
            const int acc = iter & 1;
            ok = SkWait(&st->tmemEmpty[acc], ((iter >> 1) & 1) ^ 1, st);
            if (!ok) break;
            SkFenceAfter();
            const uint32_t tmemD = tmemBase + static_cast<uint32_t>(acc * a.tn);
            for (int kb = k0; kb < k1; ++kb) {
                ok = SkWait(&st->full[stage], phase, st);
                if (!ok) break;
                SkFenceAfter();
                if (ElectOne()) {
                    const uint64_t descW = desc0 + static_cast<uint64_t>(stage * (stageBytes >> 4));
                    const uint64_t descX = descW + (GEMM_SKINNY_W_BYTES >> 4);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / GEMM_UMMA_K; ++k) {
                        SkUmma(tmemD, descW + static_cast<uint64_t>(k * 2), descX + static_cast<uint64_t>(k * 2), idesc, k != 0 || kb != k0 ? 1u : 0u);
                    }
                    SkCommit(&st->empty[stage]);
                }
                if (++stage == static_cast<uint32_t>(a.stages)) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (ok && ElectOne()) SkCommit(&st->tmemFull[acc]);
        }
    } else if (split == 1) {
        const int quad = warp & 3;                             // this warp's tensor-memory lanes: 32 output columns
        int iter = 0;
        for (int item = first; item < items; item += step, ++iter) {
            const SkinnyTile t = SkTileOf(a, item, rowStart, chunkStart, mTiles);
            const int acc = iter & 1;
            if (!SkWait(&st->tmemFull[acc], (iter >> 1) & 1, st)) break;
            SkFenceAfter();
            const int rows = min(a.tn, t.rowEnd - t.row0);
            const int n = t.n0 + quad * 32 + lane;
            for (int c0 = 0; c0 < rows; c0 += 16) {
                uint32_t r[16];
                SkTmemLoad16(tmemBase + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(acc * a.tn + c0), r);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (c0 + j < rows) SkStore(a, __uint_as_float(r[j]), n, t.row0 + c0 + j, lane);
                }
            }
            SkFenceBefore();
            __syncwarp();
            if (lane == 0) MbarArrive(&st->tmemEmpty[acc]);
        }
    } else if (first < items) {
        SkWait(&st->tmemFull[0], 0, st);                       // one item per cluster: the partial tile is complete, or given up
        SkFenceAfter();
    }

    if (split > 1) {
        // Everybody's tensor cores and loads are done with their rings: the front of every CTA's ring becomes the place where
        // it receives its slice of columns from each part, [split][tn / split][128] fp32.
        __syncthreads();
        SkClusterSync();
        const bool whole = first < items && st->abortFlag == 0;
        if (st->abortFlag != 0 && static_cast<int>(threadIdx.x) < split) {
            // this part is missing: everybody who would add it up learns so with the second barrier
            uint32_t remote;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(SmemAddr(const_cast<int *>(&st->abortFlag))), "r"(threadIdx.x));
            asm volatile("st.volatile.shared::cluster.s32 [%0], %1;" ::"r"(remote), "r"(1) : "memory");
        }
        const int slice = a.tn / split;                        // powers of two, both
        const int sliceBits = 31 - __clz(slice);
        const int quad = warp & 3;
        if (warp >= 2 && whole) {
            const uint32_t mine = SmemAddr(smem) + static_cast<uint32_t>((part * slice) * 128 + quad * 32 + lane) * 4u;
            for (int c0 = 0; c0 < a.tn; c0 += 16) {
                uint32_t r[16];
                SkTmemLoad16(tmemBase + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(c0), r);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int dst = (c0 + j) >> sliceBits;
                    uint32_t remote;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(mine + static_cast<uint32_t>(((c0 + j) & (slice - 1)) * 512)), "r"(dst));
                    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(remote), "r"(r[j]) : "memory");
                }
            }
        }
        __syncthreads();
        SkClusterSync();
        if (warp >= 2 && first < items && st->abortFlag == 0) {
            const SkinnyTile t = SkTileOf(a, first, rowStart, chunkStart, mTiles);
            const float *got = reinterpret_cast<const float *>(smem) + quad * 32 + lane;
            const int n = t.n0 + quad * 32 + lane;
            for (int i = 0; i < slice; ++i) {
                const int row = t.row0 + part * slice + i;
                if (row >= t.rowEnd) break;
                float v = got[i * 128];
                for (int s = 1; s < split; ++s) v += got[(s * slice + i) * 128];
                SkStore(a, v, n, row, lane);
            }
        }
    }

    SkFenceBefore();
    __syncthreads();
    SkFenceAfter();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(tmemCols) : "memory");
    }
    if (st->abortFlag != 0 && threadIdx.x == 0 && a.status != nullptr) atomicExch(a.status, TILEXR_DEV_MBARRIER_TIMEOUT);
}

} // namespace

const void *GemmSkinnyKernel() { return reinterpret_cast<const void *>(&TileXRGemmSkinny); }

} // namespace TileXR
