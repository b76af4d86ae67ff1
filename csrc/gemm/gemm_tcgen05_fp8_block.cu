// Block-scaled fp8 GEMM on CTA pairs (tcgen05.mma cta_group::2, kind::f8f6f4) with fp32 scales:
//
//   C[m, n] = sum over 128-wide blocks kb of  sA[m, kb] * sB[n / 128, kb] * sum_{k in kb} A[m, k] * B[n, k]
//
// A is [M, K] e4m3 with one fp32 scale per row and 128 elements of K (what the expert-parallel dispatch delivers:
// csrc/ep/ep_kernels.cu, quantisation 1 x 128), B is [N, K] e4m3 with one fp32 scale per 128 x 128 block (the usual
// weight layout beside it), C is bf16 or fp16.  fp32 scales cannot ride inside the tensor-core instruction (its
// block-scaled kinds take power-of-two E8M0 factors per 32 elements), so the sum over K is formed in two levels:
// the tensor cores produce the exact fp32 partial product of ONE 128-wide block of K into a scratch accumulator in
// tensor memory, and CUDA cores fold it into register accumulators with the block's two scales, while the tensor
// cores already work on the next block.  A stage of the TMA ring is exactly one block of K (128 bytes per row),
// so the main loop alternates two scratch accumulators:
//
//   tensor memory   2 x 256 columns: scratch p receives the pair's 256 x 256 tile for blocks of K of parity p (with
//                   cta_group::2 each CTA supplies half of B's rows: columns 0-127 and 128-255);
//   warp 0          TMA producer (this CTA's 128 rows of A and 128 rows of B per block of K, no multicast);
//   warp 1          tensor-memory owner; in the leader CTA it issues four N = 256 instructions per block of K (not two
//                   groups of N = 128, which are twice the instructions);
//   warps 2-3       idle: they complete the first warpgroup, which hands most of its registers to the others
//                   (setmaxnreg), because the promoters keep a quarter of the tile each in registers;
//   warps 4-7, 8-11 promoters of the two column halves: tcgen05.ld, scale, fused multiply-add into 128 fp32
//                   registers per thread (one row of the CTA's 128, 128 columns), release the scratch buffer as soon
//                   as its last column is in registers; at the end of a tile they round to the output type and store.
//
// What bounds a block of K: the four instructions need 512 clocks at the tensor cores' rate, the fold 128 multiply-adds per thread
// and its tensor-memory reads, and a scratch goes round through instruction, commit, fold and release, two of them in flight.
// 8192^3 with all-zero operands, where power is no limit, takes 421 us at 1965 MHz: 923 clocks per block of K, the ends of the
// tiles included (767 us with an issuer of one diverged lane, two groups of N = 128 and a scale fetched per lane and block); with
// random operands 485 - 503 us in a short loop, 569 at the power cap.
//
// Fused with the collectives of a tensor-parallel layer (mode of GemmBlockArgs):
//
//   all-gather -> GEMM    warps 2-3 of EVERY CTA, idle otherwise, write this rank's shard of A (fp8 rows and their
//                   scales) into all ranks' staging buffers, 128 rows at a time, and raise the piece's flag: through
//                   the NVLink multicast alias of the staging buffer where the runtime has one (multimem.st: one
//                   store, the switch replicates it), else with one store per peer.  No SM is set aside for
//                   communication.  The TMA warp of a CTA acquires the flag of its 128 rows before the first load of a
//                   tile (TMA then reads LOCAL memory, without multicast); each promoter warp acquires it before it
//                   reads the rows' scales.  Every rank walks the shards starting with its own, whose rows and scales it
//                   reads where they are: waiting for its own copy of them cost 90 us at 2048 x 4096 on one rank (which now takes the plain kernel).  That
//                   copy is made last, in slices of all CTAs, since nobody waits for it.
//   GEMM -> reduce-scatter    the promoters store their 128 x 256 partial tile into the row owner's staging slot and
//                   raise the tile's flag; when a CTA has run out of tiles its promoters add, in rank order, the
//                   R partial tiles of the output tiles it owns.  Every rank starts with the rows of the next rank
//                   and ends with its own.
//
// Every mbarrier wait is bounded; on a give-up all roles fall through to the tear-down, tensor memory is released
// and `status`, where the caller gives one, tells the host (the fused modes: the communicator's status).  The numerics reference is the fp32 product of the dequantised operands
// (reference numerics of the block scales: src/ep/kernels/tilexr_ep_mxfp8_quant.h:36-168 for the exponent form,
// tests/ep/demo for the 1 x 128 form).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "device/tilexr_rma.cuh"
#include "device/tilexr_sync.cuh"
#include "gemm_kernels.cuh"
#include "tilexr_types.h"

namespace TileXR {

using namespace tilexr;

namespace {

constexpr uint32_t FB_TMEM_COLS = 512;
constexpr int FB_SCRATCH = 2;               // scratch accumulators of 256 columns: two blocks of K in flight
constexpr uint32_t FB_PEER_BIT_MASK = 0xFEFFFFFFu;
constexpr int FB_HALF_N = GEMM_BN / 2;       // columns of one promoter group = one 128-wide block of the weight's scales
constexpr int FB_SEG = GEMM_FP8_BLOCK_SCALE_SEG;
constexpr int FB_SEG_PITCH = FB_SEG + 1;                  // floats per row: an odd number keeps the rows on different banks
constexpr int FB_FLAG_PLANE_A = TILEXR_FLAG_DATA_BASE;    // all-gather: piece (source rank, 128-row block) has landed
constexpr int FB_FLAG_PLANE_B = TILEXR_FLAG_ACK_BASE;     // reduce-scatter: partial tile (source rank, tile) has landed

__device__ __forceinline__ void FbMultimemSt(uint8_t *p, const Vec16 &v)
{
    asm volatile("multimem.st.relaxed.sys.global.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// `bytes` (a multiple of 16) from local memory to `dst`, four vectors per thread in flight (the pushing warps live on the 80 registers of the first warpgroup); `multicast` stores through
// an NVLink multicast address (every rank's copy at once).
__device__ __forceinline__ void FbPush(uint8_t *dst, const uint8_t *src, uint64_t bytes, int lane, int lanes, bool multicast)
{
    const uint64_t vecs = bytes / 16;
    for (uint64_t i = lane; i < vecs; i += 4ull * lanes) {
        Vec16 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t k = i + static_cast<uint64_t>(u) * lanes;
            if (k < vecs) q[u] = ld_vec16_stream(src + k * 16);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint64_t k = i + static_cast<uint64_t>(u) * lanes;
            if (k < vecs) {
                if (multicast) FbMultimemSt(dst + k * 16, q[u]);
                else st_vec16(dst + k * 16, q[u]);
            }
        }
    }
}


struct BlockState {
    uint64_t full[GEMM_FP8_BLOCK_STAGES];       // leader: both CTAs' loads of a stage have landed
    uint64_t empty[GEMM_FP8_BLOCK_STAGES];      // each CTA: the MMAs that read this stage have finished
    uint64_t scratchFull[FB_SCRATCH];      // each CTA: scratch s holds the product of one block of K
    uint64_t scratchEmpty[FB_SCRATCH];     // leader: the sixteen promoter warps of the pair have read scratch s
    uint32_t tmemBase;
    volatile int abortFlag;
    volatile int leave[2];                 // promoters: the abort flag as they all see it at the start of a segment of scales
    uint32_t epoch;                        // fused modes: the epoch of this launch (kept here, not in every thread's registers)
    float scaleB[2][2][FB_SEG];            // weight scales of the two column halves, segment by segment like the activations'
};
static_assert(sizeof(BlockState) <= 1024, "barriers and weight scales share a KB");

__device__ __forceinline__ uint32_t FbCtaRank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void FbClusterSync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t FbMapToCta(uint32_t smemAddr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smemAddr), "r"(rank));
    return r;
}
__device__ __forceinline__ int FbLoadRemoteInt(uint32_t clusterAddr)
{
    int v;
    asm volatile("ld.volatile.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(clusterAddr) : "memory");
    return v;
}
__device__ __forceinline__ void FbArriveCluster(uint32_t clusterBarAddr)
{
    // Default semantics (release at CTA scope): what the arrive has to order are this warp's tensor-memory reads, which
    // tcgen05.wait::ld and tcgen05.fence::before_thread_sync have completed; a cluster-scope release would add a
    // memory barrier to every block of K.
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(clusterBarAddr) : "memory");
}
__device__ __forceinline__ void FbTmaLoad(void *smemDst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(SmemAddr(smemDst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(SmemAddr(bar) & FB_PEER_BIT_MASK)
        : "memory");
}
__device__ __forceinline__ void FbFenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void FbFenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major operand tile written by TMA with 128-byte swizzle: rows 128 bytes apart, groups of eight rows 1024 bytes apart.
__device__ __forceinline__ uint64_t FbSmemDesc(uint32_t smemAddr)
{
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smemAddr & 0x3ffffu) >> 4);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(1024 >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}

// kind::f8f6f4, D fp32, A and B K-major, M = 256 rows over the pair, N = `width`.
__device__ __forceinline__ uint32_t FbInstrDesc(int fp8Format, int width)
{
    const uint32_t fmt = fp8Format == 2 ? 1u : 0u;
    return (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(width >> 3) << 17) | (static_cast<uint32_t>((2 * GEMM_BM) >> 4) << 24);
}

__device__ __forceinline__ void FbUmma(uint32_t tmemD, uint64_t descA, uint64_t descB, uint32_t idesc, uint32_t accumulate)
{
    const uint32_t zero = 0;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n"
        "}\n"
        ::"r"(tmemD), "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate), "r"(zero)
        : "memory");
}

// Arrives on `bar` in BOTH CTAs of the pair once every MMA issued so far has finished (an mbarrier arrive, not a load).
__device__ __forceinline__ void FbCommitPair(uint64_t *bar)
{
    const uint16_t mask = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(SmemAddr(bar)), "h"(mask) : "memory");
}

__device__ __forceinline__ void FbTmemLoad16(uint32_t taddr, uint32_t *r)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
// Waits for the loads in flight.  `r` goes through the statement: nothing else would keep the compiler from moving
// arithmetic on a load's registers in front of the wait.
__device__ __forceinline__ void FbTmemLoadWait16(uint32_t *r)
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

// A wait of this CTA has given up: neither CTA of the pair stores another tile.  A promoter that gave up goes on releasing scratch
// accumulators, which the issuer may then overwrite while the partner CTA still folds them: the partner has to know before such a
// release can be seen, hence the fence behind the store to its flag.
__device__ __forceinline__ void FbRaiseAbort(BlockState *st, uint32_t peerAbortAddr)
{
    st->abortFlag = 1;
    asm volatile("st.volatile.shared::cluster.s32 [%0], %1;\nfence.acq_rel.cluster;" ::"r"(peerAbortAddr), "r"(1) : "memory");
}

__device__ __forceinline__ bool FbWaitBar(uint64_t *bar, uint32_t parity, BlockState *st, uint32_t peerAbortAddr, uint64_t budgetNs)
{
    if (MbarTryWait(bar, parity)) return true;
    uint64_t deadline = 0;
    uint32_t polls = 0;
    for (;;) {
        if (MbarTryWait(bar, parity)) return true;
        if ((++polls & 127u) == 0) {
            if (st->abortFlag != 0 || FbLoadRemoteInt(peerAbortAddr) != 0) {
                FbRaiseAbort(st, peerAbortAddr);
                return false;
            }
            const uint64_t t = now_ns();
            if (deadline == 0) {
                deadline = t + budgetNs;
            } else if (t > deadline) {
                FbRaiseAbort(st, peerAbortAddr);
                return false;
            }
        }
    }
}

// The same by a whole warp, with one verdict for all lanes.
__device__ __forceinline__ bool FbWaitBarWarp(uint64_t *bar, uint32_t parity, BlockState *st, uint32_t peerAbortAddr, uint64_t budgetNs)
{
    return __all_sync(0xffffffffu, FbWaitBar(bar, parity, st, peerAbortAddr, budgetNs)) != 0;
}

// Bounded acquire of a flag by one thread that has no Waiter of its own (the promoters are short of registers).
__device__ __forceinline__ bool FbAcquireFlag(const uint64_t *flag, uint64_t want, BlockState *st, uint64_t budgetNs)
{
    uint64_t deadline = 0;
    uint32_t polls = 0;
    while (ld_acquire_sys_u64(flag) < want) {
        if ((++polls & 63u) == 0) {
            if (st->abortFlag != 0) return false;
            const uint64_t t = now_ns();
            if (deadline == 0) {
                deadline = t + budgetNs;
            } else if (t > deadline) {
                st->abortFlag = 1;
                return false;
            }
        }
    }
    return true;
}

__device__ __forceinline__ uint32_t FbPackPair(float lo, float hi, bool bf16)
{
    if (bf16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t *>(&v);
    }
    const __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// acc[0, 1] += x[0, 1] * f in one instruction, each rounded like fmaf.
__device__ __forceinline__ void FbFma2(const uint32_t *x, float f, float *acc)
{
    asm("{\n"
        ".reg .b64 xx, ff, aa;\n"
        "mov.b64 xx, {%2, %3};\n"
        "mov.b64 ff, {%4, %4};\n"
        "mov.b64 aa, {%0, %1};\n"
        "fma.rn.f32x2 aa, xx, ff, aa;\n"
        "mov.b64 {%0, %1}, aa;\n"
        "}\n"
        : "+f"(acc[0]), "+f"(acc[1])
        : "r"(x[0]), "r"(x[1]), "f"(f));
}

// The grouped tile walk of the bf16 CTA-pair kernel: 256-row blocks advance fastest inside a group.
__device__ __forceinline__ void FbTileAt(int t, int mTiles, int nBlocks, int GROUP, int *mTile, int *nBlock)
{
    const int perGroup = GROUP * nBlocks;
    const int group = t / perGroup;
    const int first = group * GROUP;
    const int size = min(GROUP, mTiles - first);
    const int u = t - group * perGroup;
    *mTile = first + u % size;
    *nBlock = u / size;
}

// Tile t of this pair's walk.  In the fused modes the 256-row blocks are rotated so that every rank starts with its own
// shard (all-gather: its rows are there first) or with the next rank's (reduce-scatter: its own rows come last, when the
// peers' partial tiles have had time to arrive).
__device__ __forceinline__ void FbTileOf(const GemmBlockArgs &a, int t, int mTiles, int rank, int *mTile, int *nBlock)
{
    FbTileAt(t, mTiles, a.nBlocks, a.rasterGroup, mTile, nBlock);
    if (a.mode != GEMM_PLAIN) {
        const int pairsPerShard = a.blocksPerShard / 2;
        const int first = (a.mode == GEMM_ALL_GATHER ? rank : rank + 1) * pairsPerShard;
        *mTile = (*mTile + first) % mTiles;
    }
}

template <int N> struct FbCols { static constexpr int value = N; };

struct FbItem {
    int mTile, nBlock;
    int col0, width;     // columns of C
};

// Item `i` of the launch: a whole tile or, in the plain mode, a slice of one.  A slice may lie past the last column (col0 >= N): nobody works on it.
template <int MODE>
__device__ __forceinline__ FbItem FbItemOf(const GemmBlockArgs &a, int i, int mTiles, int rank)
{
    FbItem it;
    int t = i, slice = 0;
    it.width = GEMM_BN;
    if (MODE == GEMM_PLAIN && i >= a.wideTiles) {
        const int per = GEMM_BN / a.sliceWidth;
        const int u = i - a.wideTiles;
        t = a.wideTiles + u / per;
        slice = u % per;
        it.width = a.sliceWidth;
    }
    FbTileOf(a, t, mTiles, rank, &it.mTile, &it.nBlock);
    it.col0 = it.nBlock * GEMM_BN + slice * it.width;
    return it;
}

// Twelve warps start with 168 registers each (the most a block of this size can have); the first warpgroup then
// shrinks to 80 and the two promoter warpgroups grow to 208 (128 x 80 + 256 x 208 of the 384 x 168 registers of the launch),
// so that 128 accumulators and two 16-register tensor-memory reads fit.
// One kernel per mode: with the collectives' code in it the plain kernel spilled inside the fold (8192^3: 511 us with it, 474 us without).
template <int MODE>
__device__ __forceinline__ void FbBody(const GemmBlockArgs &a)
{
    extern __shared__ uint8_t smemRaw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint8_t *stageBase = smem;
    BlockState *st = reinterpret_cast<BlockState *>(smem + GEMM_FP8_BLOCK_STAGES * GEMM_PAIR_STAGE_BYTES);
    uint8_t *scales = smem + GEMM_FP8_BLOCK_STAGES * GEMM_PAIR_STAGE_BYTES + 1024;      // two buffers of 128 rows' scales
    uint8_t *stageC = scales + 2 * GEMM_FP8_BLOCK_SCALES_BYTES;                         // the promoter warps' staging tiles

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t ctaRank = FbCtaRank();
    const bool leader = ctaRank == 0;
    constexpr bool fused = MODE != GEMM_PLAIN;
    const uint32_t peerAbortAddr = FbMapToCta(SmemAddr(const_cast<int *>(&st->abortFlag)), ctaRank ^ 1u);

    // The promoters have no register to spare for values that only the prologue, the TMA lane and the epilogue need: the
    // launch's epoch lives in shared memory, and rank, rank count and the wait budget are read where they are used.
    bool ok = true;
    if (fused) {
        // The staging buffers are not double buffered: nobody writes into a peer's before that peer has finished the
        // previous launch on this communicator.
        Waiter w = MakeWaiter(a.comm, a.magic, blockIdx.x);
        const int rank = a.comm->rank;
        const int ranks = a.comm->rankSize;
        if (threadIdx.x == 0) st->epoch = w.epoch;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.comm->dfx[TILEXR_DFX_MAGIC] = w.epoch;
            a.comm->dfx[TILEXR_DFX_OP] = MODE == GEMM_ALL_GATHER ? TILEXR_OP_ALL_GATHER_MATMUL : TILEXR_OP_MATMUL_REDUCE_SCATTER;
            a.comm->dfx[TILEXR_DFX_RUN_STATUS] = TILEXR_RUN_STARTED;
        }
        bool g = true;
        if (w.epoch >= 2 && static_cast<int>(threadIdx.x) < ranks && static_cast<int>(threadIdx.x) != rank) {
            g = WaitPeerFinished(w, threadIdx.x, w.epoch - 1);
        }
        ok = BlockBroadcastOk(g);
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < GEMM_FP8_BLOCK_STAGES; ++s) {
            MbarInit(&st->full[s], 1);
            MbarInit(&st->empty[s], 1);
        }
        for (int h = 0; h < FB_SCRATCH; ++h) {
            MbarInit(&st->scratchFull[h], 1);     // one commit
            MbarInit(&st->scratchEmpty[h], 16);   // eight promoter warps in each of the two CTAs
        }
        st->abortFlag = ok ? 0 : 1;
        MbarInitFence();
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&a.tmapA)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&a.tmapB)) : "memory");
    }
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(SmemAddr(&st->tmemBase)), "r"(FB_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    StreamRelease();
    StreamWait();
    FbFenceBefore();
    __syncthreads();
    FbClusterSync();
    FbFenceAfter();
    const uint32_t tmemBase = st->tmemBase;

    const int mTiles = (a.M + 2 * GEMM_BM - 1) / (2 * GEMM_BM);
    const int items = a.items;
    const int pair = static_cast<int>(blockIdx.x) >> 1;
    const int nPairs = static_cast<int>(gridDim.x) >> 1;
    const bool bf16 = a.isBf16 != 0;

    if (warp < 4) {
    // the first warpgroup gives registers away (all four warps execute this together) and then splits into its roles
    asm volatile("setmaxnreg.dec.sync.aligned.u32 80;" ::: "memory");
    if (warp == 0) {
        // ---- TMA producer (the warp runs whole and elects a lane to issue, see ElectOne) ----------------------------
        const uint64_t budgetNs = fused ? a.comm->waitTimeoutNs : 4000000000ull;
        const int rank = fused ? a.comm->rank : 0;
        Waiter w{fused ? a.comm : nullptr, st->epoch, static_cast<int32_t>(blockIdx.x), TILEXR_DEV_OK, 0};
        uint32_t stage = 0, phase = 0;
        for (int t = pair; t < items && __all_sync(0xffffffffu, st->abortFlag == 0); t += nPairs) {
            const FbItem it = FbItemOf<MODE>(a, t, mTiles, rank);
            if (it.col0 >= a.N) continue;
            const int rowA = it.mTile * 2 * GEMM_BM + static_cast<int>(ctaRank) * GEMM_BM;
            const int rowB = it.col0 + static_cast<int>(ctaRank) * (it.width / 2);       // each CTA supplies half of the item's rows of B
            const uint32_t stageBytes = GEMM_STAGE_A_BYTES + static_cast<uint32_t>(it.width / 2) * 128u;
            bool own = false;              // the rows are this rank's shard
            if (MODE == GEMM_ALL_GATHER) {
                // this CTA's 128 rows of the gathered A: wait until their owner has written them here
                const int block = rowA / GEMM_BM;
                const int shard = block / a.blocksPerShard;
                const int64_t slot = FB_FLAG_PLANE_A + static_cast<int64_t>(shard) * a.flagStride + (block - shard * a.blocksPerShard);
                bool landed = true;
                own = shard == rank;
                if (lane == 0 && !own) landed = WaitFlagGE(w, FlagSlot(a.comm, rank, slot), 1, shard, slot);
                if (!__all_sync(0xffffffffu, landed)) {
                    st->abortFlag = 1;
                    break;
                }
                __syncwarp();              // the rows lane 0 acquired are there for the lane that issues
                fence_proxy_async();       // the rows were written by generic-proxy stores, TMA reads them next
            }
            const CUtensorMap *mapA = own ? &a.tmapALocal : &a.tmapA;
            const int yA = own ? rowA - rank * a.shardRows : rowA;
            bool broke = false;
            for (int kb = 0; kb < a.kBlocks; ++kb) {
                if (!FbWaitBarWarp(&st->empty[stage], phase ^ 1u, st, peerAbortAddr, budgetNs)) {
                    broke = true;
                    break;
                }
                if (ElectOne()) {
                    uint8_t *sa = stageBase + stage * GEMM_PAIR_STAGE_BYTES;
                    uint8_t *sb = sa + GEMM_STAGE_A_BYTES;
                    if (leader) MbarExpectTx(&st->full[stage], 2 * stageBytes);
                    FbTmaLoad(sa, mapA, kb * 128, yA, &st->full[stage]);       // x in bytes = elements: a multiple of 128
                    if (MODE != GEMM_PLAIN || it.width == GEMM_BN) {
                        FbTmaLoad(sb, &a.tmapB, kb * 128, rowB, &st->full[stage]);
                    } else {
                        for (int r = 0; r < it.width / 2; r += GEMM_FP8_SLICE_BOX) FbTmaLoad(sb + r * 128, &a.tmapBSlice, kb * 128, rowB + r, &st->full[stage]);
                    }
                }
                if (++stage == GEMM_FP8_BLOCK_STAGES) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (broke) break;
        }
    } else if (warp == 1) {
        // ---- MMA issuer: per block of K, four N = 256 instructions into the scratch of its parity --------------------
        if (leader) {
            const uint64_t budgetNs = fused ? a.comm->waitTimeoutNs : 4000000000ull;
            const uint64_t descA0 = FbSmemDesc(SmemAddr(stageBase));
            const uint64_t descB0 = FbSmemDesc(SmemAddr(stageBase) + GEMM_STAGE_A_BYTES);
            uint32_t stage = 0, phase = 0;
            uint32_t kbAll = 0;                    // blocks of K issued so far, over all tiles: the scratch buffers alternate with it
            for (int t = pair; t < items && __all_sync(0xffffffffu, st->abortFlag == 0); t += nPairs) {
                const FbItem it = FbItemOf<MODE>(a, t, mTiles, 0);       // its width and whether it exists, the same for every rank
                if (it.col0 >= a.N) continue;
                const uint32_t idesc = FbInstrDesc(a.fp8Format, it.width);
                bool broke = false;
                for (int kb = 0; kb < a.kBlocks; ++kb, ++kbAll) {
                    const uint32_t p = kbAll & 1u;
                    if (!FbWaitBarWarp(&st->full[stage], phase, st, peerAbortAddr, budgetNs) ||
                        !FbWaitBarWarp(&st->scratchEmpty[p], ((kbAll >> 1) & 1u) ^ 1u, st, peerAbortAddr, budgetNs)) {
                        broke = true;
                        break;
                    }
                    FbFenceAfter();
                    if (ElectOne()) {
                        const uint64_t descA = descA0 + static_cast<uint64_t>(stage * (GEMM_PAIR_STAGE_BYTES >> 4));
                        const uint64_t descB = descB0 + static_cast<uint64_t>(stage * (GEMM_PAIR_STAGE_BYTES >> 4));
                        const uint32_t tmemD = tmemBase + p * GEMM_BN;
#pragma unroll
                        for (int k = 0; k < 4; ++k) {       // 32 elements of K (32 bytes) per instruction: +2 descriptor units
                            FbUmma(tmemD, descA + static_cast<uint64_t>(k * 2), descB + static_cast<uint64_t>(k * 2), idesc, k != 0 ? 1u : 0u);
                        }
                        FbCommitPair(&st->scratchFull[p]);
                        FbCommitPair(&st->empty[stage]);
                    }
                    if (++stage == GEMM_FP8_BLOCK_STAGES) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (broke) break;
            }
        }
    } else if (MODE == GEMM_ALL_GATHER && ok) {
        // ---- warps 2-3: write this rank's shard, rows and scales, into every rank's staging buffers -------------------
        const int pt2 = static_cast<int>(threadIdx.x) - 64;           // 0..63
        const int rank = a.comm->rank, ranks = a.comm->rankSize;
        const uint32_t epoch = st->epoch;
        const TileXRRegistry *reg = a.comm->registryPtr;
        uint8_t *mcRows = reg->regions[a.aHandle].mcBase;
        uint8_t *mcScales = reg->regions[a.sHandle].mcBase;
        const bool multicast = ranks > 1 && mcRows != nullptr && mcScales != nullptr;
        const int pieces = a.blocksPerShard;
        const int items = multicast ? pieces : (ranks - 1) * pieces;
        const uint64_t rowBytes = static_cast<uint64_t>(a.K);
        const uint64_t scaleRowBytes = static_cast<uint64_t>(a.kBlocks) * 4;
        for (int it = blockIdx.x; it < items; it += gridDim.x) {
            const int piece = it % pieces;
            const int peer = (rank - 1 - it / pieces + ranks) % ranks;      // rank-1 needs it first
            const uint64_t srcRow = static_cast<uint64_t>(piece) * GEMM_BM;
            const uint64_t dstRow = static_cast<uint64_t>(rank) * a.shardRows + srcRow;
            uint8_t *rowsTo = (multicast ? mcRows : reg->regions[a.aHandle].peerBase[peer]) + a.aOffset + dstRow * rowBytes;
            uint8_t *scalesTo = (multicast ? mcScales : reg->regions[a.sHandle].peerBase[peer]) + a.sOffset + dstRow * scaleRowBytes;
            FbPush(rowsTo, a.aLocal + srcRow * rowBytes, GEMM_BM * rowBytes, pt2, 64, multicast);
            FbPush(scalesTo, reinterpret_cast<const uint8_t *>(a.scaleALocal) + srcRow * scaleRowBytes, GEMM_BM * scaleRowBytes, pt2, 64, multicast);
            asm volatile("bar.sync 2, 64;" ::: "memory");
            if (pt2 == 0) {
                fence_acq_rel_sys();
                const uint64_t up = MakeFlag(epoch, 1);
                const int64_t slot = FB_FLAG_PLANE_A + static_cast<int64_t>(rank) * a.flagStride + piece;
                if (multicast) {
                    for (int r = 0; r < ranks; ++r) st_relaxed_sys_u64(FlagSlot(a.comm, r, slot), up);
                } else {
                    st_relaxed_sys_u64(FlagSlot(a.comm, peer, slot), up);
                }
            }
            asm volatile("bar.sync 2, 64;" ::: "memory");
        }
        if (!multicast) {
            // the caller finds all rows in its staging buffers, its own among them: a slice of them per CTA, no flags
            auto slice = [&](uint8_t *dst, const uint8_t *src, uint64_t bytes) {
                const uint64_t per = ((bytes / 16 + gridDim.x - 1) / gridDim.x) * 16;
                const uint64_t b0 = min(bytes, per * blockIdx.x);
                FbPush(dst + b0, src + b0, min(bytes - b0, per), pt2, 64, false);
            };
            const uint64_t myRow = static_cast<uint64_t>(rank) * a.shardRows;
            slice(reg->regions[a.aHandle].peerBase[rank] + a.aOffset + myRow * rowBytes, a.aLocal, a.shardRows * rowBytes);
            slice(reg->regions[a.sHandle].peerBase[rank] + a.sOffset + myRow * scaleRowBytes, reinterpret_cast<const uint8_t *>(a.scaleALocal),
                  a.shardRows * scaleRowBytes);
        }
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 208;" ::: "memory");
        // ---- promoters: warps 4-7 own column half 0, warps 8-11 half 1; TMEM lanes 32 * (warp % 4) .. + 31 --------------
        const int quad = warp & 3;
        const int h = (warp - 4) >> 2;
        const int myRow = quad * 32 + lane;                       // row of this CTA's 128-row sub-tile
        const int pt = static_cast<int>(threadIdx.x) - 128;       // 0..255 among the promoter threads
        uint8_t *myStage = stageC + (warp - 4) * (32 * 128);
        uint32_t kbAll = 0;                        // as the issuer counts it: scratch kbAll & 1, its (kbAll >> 1)-th use
        const int KB = a.kBlocks;
        const int segments = (KB + FB_SEG - 1) / FB_SEG;
        const int segBlocks = (KB + segments - 1) / segments;
        const bool gathered = MODE == GEMM_ALL_GATHER;
        const uint64_t budgetNs = fused ? a.comm->waitTimeoutNs : 4000000000ull;
        auto ofPeer = [&](int mTile) {
            const int64_t row = static_cast<int64_t>(mTile) * 2 * GEMM_BM + static_cast<int64_t>(ctaRank) * GEMM_BM;
            return gathered && row / a.shardRows != a.comm->rank;
        };
        // Brings the scales of an item, blocks kb0 .. kb0 + segBlocks - 1 of K, to buffer `buf`: of this CTA's 128 rows, a warp takes a row
        // at a time, and of the two column halves.  Scales that a peer writes during this launch are read through L2, never through the
        // read-only path.
        auto loadScales = [&](const FbItem &it, bool fromPeer, int kb0, uint32_t buf) {
            const int64_t tileRow = static_cast<int64_t>(it.mTile) * 2 * GEMM_BM + static_cast<int64_t>(ctaRank) * GEMM_BM;
            const float *sa = a.scaleA + tileRow * KB;
            if (gathered && !fromPeer) sa = a.scaleALocal + (tileRow - static_cast<int64_t>(a.comm->rank) * a.shardRows) * KB;
            const int rows = static_cast<int>(min(static_cast<int64_t>(GEMM_BM), a.M - tileRow));
            const int n = min(segBlocks, KB - kb0);
            float *to = reinterpret_cast<float *>(scales + buf * GEMM_FP8_BLOCK_SCALES_BYTES);
            if (lane < n) {
#pragma unroll 4
                for (int r = pt >> 5; r < rows; r += 8) {
                    const float *src = sa + static_cast<int64_t>(r) * KB + kb0 + lane;
                    float *dst = to + r * FB_SEG_PITCH + lane;
                    if (fromPeer) *dst = __ldcg(src);
                    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(SmemAddr(dst)), "l"(src) : "memory");
                }
                if (pt < 64) {
                    const int block = min((it.col0 + (pt >> 5) * (it.width / 2)) / FB_HALF_N, a.scaleBRows - 1);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(SmemAddr(&st->scaleB[buf][pt >> 5][lane])),
                                 "l"(a.scaleB + static_cast<int64_t>(block) * KB + kb0 + lane) : "memory");
                }
            }
        };
        uint32_t seg = 0;                          // segments so far: the scales' buffers alternate with it
        bool ahead = false;                        // the segment's scales are already on their way
        FbItem nextItem;
        int nextT = pair;
        auto findItem = [&] {                      // the next item that exists
            for (; nextT < items; nextT += nPairs) {
                nextItem = FbItemOf<MODE>(a, nextT, mTiles, fused ? a.comm->rank : 0);
                if (nextItem.col0 < a.N) return;
            }
        };
        // One item, of which this thread folds COLS columns of its row.  False: a wait has given up, nobody goes on.
        auto foldItem = [&](auto tag, const FbItem &it) -> bool {
            constexpr int COLS = decltype(tag)::value;
            const bool fromPeer = ofPeer(it.mTile);
            if (fromPeer) {
                // the scales of these 128 rows were written by their owner during this launch: acquire the rows' flag first
                if (lane == 0) {
                    const int block = it.mTile * 2 + static_cast<int>(ctaRank);
                    const int shard = block / a.blocksPerShard;
                    const int64_t slot = FB_FLAG_PLANE_A + static_cast<int64_t>(shard) * a.flagStride + (block - shard * a.blocksPerShard);
                    FbAcquireFlag(FlagSlot(a.comm, a.comm->rank, slot), MakeFlag(st->epoch, 1), st, budgetNs);
                }
                __syncwarp();
            }
            float acc[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) acc[j] = 0.f;
            for (int kb0 = 0; kb0 < KB; kb0 += segBlocks, ++seg) {
                // The scales go through shared memory: a lane reading its own row's scale from memory for every block touches 32 lines per warp
                // and block.  Those of the next segment, of this item or the next one, come while this one is folded: fetched between
                // two items they, and the stores of a row per lane, took 7.8 us of every tile (2.4 now).
                const uint32_t buf = seg & 1u;
                if (!ahead) loadScales(it, fromPeer, kb0, buf);
                asm volatile("cp.async.wait_all;" ::: "memory");
                if (pt == 0) st->leave[buf] = st->abortFlag;
                asm volatile("bar.sync 1, 256;" ::: "memory");      // this segment's scales are there, the one before has been read
                if (st->leave[buf] != 0) return false;              // all eight warps together: none may miss a barrier
                if (kb0 + segBlocks < KB) {
                    ahead = !fromPeer;
                    if (ahead) loadScales(it, false, kb0 + segBlocks, buf ^ 1u);
                } else {
                    nextT += nPairs;
                    findItem();
                    ahead = nextT < items && !ofPeer(nextItem.mTile);
                    if (ahead) loadScales(nextItem, false, 0, buf ^ 1u);
                }
                const float *sa = reinterpret_cast<const float *>(scales + buf * GEMM_FP8_BLOCK_SCALES_BYTES) + myRow * FB_SEG_PITCH;
                const float *sb = st->scaleB[buf][h];
                const int n = min(segBlocks, KB - kb0);
                // One way in and one way out: with an exit for a wait that gave up, the 128 accumulators were moved to other
                // registers and back in every block.  Such a wait has raised the abort flag of both CTAs; what either folds after
                // it is never stored (a test of the verdict in front of the release cost 2 %).
                for (int kb = 0; kb < n; ++kb) {
                    const float f = sa[kb] * sb[kb];
                    const uint32_t p = kbAll & 1u;
                    FbWaitBarWarp(&st->scratchFull[p], (kbAll >> 1) & 1u, st, peerAbortAddr, budgetNs);
                    ++kbAll;
                    FbFenceAfter();
                    const uint32_t taddr = tmemBase + (static_cast<uint32_t>(quad * 32) << 16) + p * GEMM_BN + static_cast<uint32_t>(h * COLS);
                    // Sixteen columns at a time, the next ones on their way while these are folded.  In a whole tile one column per multiply-add:
                    // two are quicker by themselves (285 clocks per block, 351 with one) but slow down beside the tensor cores, which read and
                    // write the same memory (608 and 371): 8192^3 564 us and 514 to 548, 2048 x 14336 x 4096 128 and 120.  A narrow one leaves
                    // the tensor cores idle anyway: 600 x 2048 x 8192 29.5 us and, one column at a time, 32.
                    uint32_t r[2][16];
                    FbTmemLoad16(taddr, r[0]);
#pragma unroll
                    for (int cc = 0; cc < COLS / 16; ++cc) {
                        FbTmemLoadWait16(r[cc & 1]);
                        if (cc < COLS / 16 - 1) {
                            FbTmemLoad16(taddr + (cc + 1) * 16, r[(cc + 1) & 1]);
                        } else {
                            // the columns are in registers: the issuer may overwrite them two blocks of K from now
                            FbFenceBefore();
                            __syncwarp();
                            if (lane == 0) FbArriveCluster(SmemAddr(&st->scratchEmpty[p]) & FB_PEER_BIT_MASK);
                        }
                        float *to = acc + cc * 16;
                        if constexpr (COLS == FB_HALF_N) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) to[j] = fmaf(__uint_as_float(r[cc & 1][j]), f, to[j]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; j += 2) FbFma2(r[cc & 1] + j, f, to + j);
                        }
                    }
                }
            }
            // What a wait that gave up has spoilt is not stored: its warp raised the flag before it released the scratch, so every warp that
            // folded what came after sees it here.
            const bool whole = __all_sync(0xffffffffu, st->abortFlag == 0) != 0;
            const int64_t row0 = static_cast<int64_t>(it.mTile) * 2 * GEMM_BM + static_cast<int64_t>(ctaRank) * GEMM_BM;
            uint8_t *base;                         // row `row0` of C, or of its owner's staging slot for this rank
            int rows = GEMM_BM;
            int owner = 0, tileLocal = 0;
            if (MODE == GEMM_REDUCE_SCATTER) {
                const int block = static_cast<int>(row0 / GEMM_BM);
                owner = block / a.blocksPerShard;
                const int localBlock = block - owner * a.blocksPerShard;
                tileLocal = localBlock * a.nBlocks + it.nBlock;
                base = a.comm->registryPtr->regions[a.outHandle].peerBase[owner] + a.outOffset +
                       (static_cast<uint64_t>(a.comm->rank) * a.shardRows + static_cast<uint64_t>(localBlock) * GEMM_BM) * a.N * 2;
            } else {
                base = a.c + static_cast<uint64_t>(row0) * a.N * 2;
                rows = static_cast<int>(min(static_cast<int64_t>(GEMM_BM), a.M - row0));
            }
            // Through a staging tile of the warp's own, 32 rows by 64 columns, so that a warp stores whole lines: a row per lane is 32 lines per
            // instruction.
            if (whole) {
                constexpr int CHUNKS = (COLS < 64 ? COLS : 64) / 8;      // 16-byte chunks of a row per round
#pragma unroll
                for (int round = 0; round < COLS / (CHUNKS * 8); ++round) {
                    __syncwarp();
#pragma unroll
                    for (int v = 0; v < CHUNKS; ++v) {
                        uint32_t w[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            w[j] = FbPackPair(acc[(round * CHUNKS + v) * 8 + 2 * j], acc[(round * CHUNKS + v) * 8 + 2 * j + 1], bf16);
                        }
                        *reinterpret_cast<uint4 *>(myStage + lane * 128 + ((v ^ (lane & 7)) * 16)) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                    __syncwarp();
                    const int colRound = it.col0 + h * COLS + round * CHUNKS * 8;
#pragma unroll
                    for (int k = 0; k < CHUNKS; ++k) {
                        const int idx = k * 32 + lane;
                        const int rr = idx / CHUNKS, ch = idx % CHUNKS;
                        const int col = colRound + ch * 8;
                        if (quad * 32 + rr < rows && col < a.N) {
                            const uint4 v = *reinterpret_cast<const uint4 *>(myStage + rr * 128 + ((ch ^ (rr & 7)) * 16));
                            st_vec16(base + static_cast<uint64_t>(quad * 32 + rr) * a.N * 2 + static_cast<uint64_t>(col) * 2, Vec16{v.x, v.y, v.z, v.w});
                        }
                    }
                }
            }
            if (MODE == GEMM_REDUCE_SCATTER) {
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (pt == 0 && st->abortFlag == 0) {
                    // all 256 promoter threads have stored (the barrier above): order their stores, then tell the owner
                    fence_acq_rel_sys();
                    st_relaxed_sys_u64(FlagSlot(a.comm, owner, FB_FLAG_PLANE_B + static_cast<int64_t>(a.comm->rank) * a.flagStride + tileLocal),
                                       MakeFlag(st->epoch, 1));
                }
            }
            return true;
        };
        findItem();
        for (bool go = true; go && nextT < items;) {
            const FbItem it = nextItem;
            if (MODE != GEMM_PLAIN || it.width == GEMM_BN) go = foldItem(FbCols<FB_HALF_N>{}, it);
            else if (it.width == 128) go = foldItem(FbCols<64>{}, it);
            else if (it.width == 64) go = foldItem(FbCols<32>{}, it);
            else go = foldItem(FbCols<16>{}, it);
        }
        // ---- reduce-scatter: add the partial tiles of the output tiles this CTA owns, in rank order ---------------------
        if (MODE == GEMM_REDUCE_SCATTER) {
            const int owned = a.blocksPerShard * a.nBlocks;
            const int rank = a.comm->rank, ranks = a.comm->rankSize;
            const uint32_t epoch = st->epoch;
            const uint8_t *stage = a.comm->registryPtr->regions[a.outHandle].peerBase[rank] + a.outOffset;
            const uint64_t rowBytes = static_cast<uint64_t>(a.N) * 2;
            for (int tl = static_cast<int>(blockIdx.x); tl < owned; tl += static_cast<int>(gridDim.x)) {
                asm volatile("bar.sync 1, 256;" ::: "memory");          // the word of the previous round has been read
                if (pt == 0) st->leave[0] = st->abortFlag;
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (st->leave[0] != 0) break;
                if (pt < ranks) {
                    const int64_t slot = FB_FLAG_PLANE_B + static_cast<int64_t>(pt) * a.flagStride + tl;
                    FbAcquireFlag(FlagSlot(a.comm, rank, slot), MakeFlag(epoch, 1), st, budgetNs);
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (st->abortFlag != 0) continue;                       // uniform after the barrier: the next round leaves
                const int mLocal = tl / a.nBlocks;
                const int nBlock = tl % a.nBlocks;
                const int cols = min(GEMM_BN, a.N - nBlock * GEMM_BN);
                const int vecsPerRow = cols / 8;
                const int total = GEMM_BM * vecsPerRow;
                for (int i0 = pt; i0 < total; i0 += 256 * 2) {
                    float accv[2][8];
                    uint64_t off[2];
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int i = min(i0 + q * 256, total - 1);
                        off[q] = (static_cast<uint64_t>(mLocal) * GEMM_BM + i / vecsPerRow) * rowBytes +
                                 (static_cast<uint64_t>(nBlock) * GEMM_BN + (i % vecsPerRow) * 8) * 2;
                    }
                    for (int s = 0; s < ranks; ++s) {
                        Vec16 x[2];
#pragma unroll
                        for (int q = 0; q < 2; ++q) x[q] = ld_vec16_stream(stage + static_cast<uint64_t>(s) * a.shardRows * rowBytes + off[q]);
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const uint32_t wds[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                float lo, hi;
                                if (bf16) {
                                    lo = __uint_as_float(wds[j] << 16);
                                    hi = __uint_as_float(wds[j] & 0xffff0000u);
                                } else {
                                    const float2 f2 = __half22float2(*reinterpret_cast<const __half2 *>(&wds[j]));
                                    lo = f2.x;
                                    hi = f2.y;
                                }
                                accv[q][2 * j] = s == 0 ? lo : accv[q][2 * j] + lo;
                                accv[q][2 * j + 1] = s == 0 ? hi : accv[q][2 * j + 1] + hi;
                            }
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        if (i0 + q * 256 < total) {
                            st_vec16(a.c + off[q], Vec16{FbPackPair(accv[q][0], accv[q][1], bf16), FbPackPair(accv[q][2], accv[q][3], bf16),
                                                         FbPackPair(accv[q][4], accv[q][5], bf16), FbPackPair(accv[q][6], accv[q][7], bf16)});
                        }
                    }
                }
            }
        }
    }

    // ---- tear-down -------------------------------------------------------------------------------------------------------
    FbFenceBefore();
    __syncthreads();
    FbClusterSync();
    FbFenceAfter();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmemBase), "r"(FB_TMEM_COLS) : "memory");
    }
    const bool failed = st->abortFlag != 0;
    if (failed && threadIdx.x == 0 && a.status != nullptr) atomicExch(a.status, TILEXR_DEV_MBARRIER_TIMEOUT);
    if (fused) {
        Waiter w{a.comm, st->epoch, static_cast<int32_t>(blockIdx.x), TILEXR_DEV_OK, 0};
        if (failed && threadIdx.x == 0) RaiseFailure(w, TILEXR_DEV_MBARRIER_TIMEOUT, a.comm->rank, blockIdx.x, 0, 0);
        KernelEpilogue(w, !failed);
    }
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_FP8_BLOCK_THREADS, 1)
TileXRGemmFp8BlockScaled(const __grid_constant__ GemmBlockArgs a) { FbBody<MODE>(a); }
// Emulated worlds: one argument block per rank in global memory, rank = blockIdx.y.
template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_FP8_BLOCK_THREADS, 1)
TileXRGemmFp8BlockScaled_emulated(const GemmBlockArgs *perRank) { FbBody<MODE>(perRank[blockIdx.y]); }

// Two pieces of memory, 16-byte vectors, four in flight per thread.
__global__ void __launch_bounds__(256) TileXRStageCopy(uint8_t *dst0, const uint8_t *src0, int64_t vecs0, uint8_t *dst1, const uint8_t *src1, int64_t vecs1)
{
    StreamRelease();
    StreamWait();
    const int64_t threads = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i0 = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < vecs0 + vecs1; i0 += 4 * threads) {
        Vec16 q[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = i0 + u * threads;
            if (i < vecs0 + vecs1) q[u] = ld_vec16_stream(i < vecs0 ? src0 + i * 16 : src1 + (i - vecs0) * 16);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int64_t i = i0 + u * threads;
            if (i < vecs0 + vecs1) st_vec16(i < vecs0 ? dst0 + i * 16 : dst1 + (i - vecs0) * 16, q[u]);
        }
    }
}

} // namespace

const void *StageCopyKernel() { return reinterpret_cast<const void *>(&TileXRStageCopy); }
const void *GemmFp8BlockKernel(int mode)
{
    return mode == GEMM_ALL_GATHER       ? reinterpret_cast<const void *>(&TileXRGemmFp8BlockScaled<GEMM_ALL_GATHER>)
           : mode == GEMM_REDUCE_SCATTER ? reinterpret_cast<const void *>(&TileXRGemmFp8BlockScaled<GEMM_REDUCE_SCATTER>)
                                         : reinterpret_cast<const void *>(&TileXRGemmFp8BlockScaled<GEMM_PLAIN>);
}
const void *GemmFp8BlockKernelEmulated(int mode)
{
    return mode == GEMM_ALL_GATHER ? reinterpret_cast<const void *>(&TileXRGemmFp8BlockScaled_emulated<GEMM_ALL_GATHER>)
                                   : reinterpret_cast<const void *>(&TileXRGemmFp8BlockScaled_emulated<GEMM_REDUCE_SCATTER>);
}

} // namespace TileXR
