// Argument block of the tcgen05 GEMM family (plain, all-gather -> GEMM, GEMM -> reduce-scatter).
#ifndef TILEXR_GEMM_KERNELS_CUH
#define TILEXR_GEMM_KERNELS_CUH

#include <cuda.h>
#include <stdint.h>

#include "gemm_few_rows.h"
#include "tilexr_comm_args.h"
#include "tilexr_launch.h"

namespace TileXR {

constexpr int GEMM_BM = 128;        // rows of C per tile  = UMMA M
constexpr int GEMM_BN = 256;        // columns of C per tile = UMMA N
constexpr int GEMM_BK = 64;         // K per pipeline stage = one 128-byte swizzle row of bf16
constexpr int GEMM_UMMA_K = 16;     // K of one tcgen05.mma for 16-bit inputs
constexpr int GEMM_STAGES = 4;
constexpr unsigned GEMM_THREADS = 192;   // warp 0: TMA, warp 1: MMA + TMEM owner, warps 2-5: epilogue
constexpr unsigned GEMM_PAIR_THREADS = 256;   // CTA-pair kernel: two more warps that push this rank's shard in the all-gather mode
constexpr uint32_t GEMM_STAGE_A_BYTES = GEMM_BM * GEMM_BK * 2;
constexpr uint32_t GEMM_STAGE_B_BYTES = GEMM_BN * GEMM_BK * 2;
constexpr uint32_t GEMM_STAGE_BYTES = GEMM_STAGE_A_BYTES + GEMM_STAGE_B_BYTES;
constexpr size_t GEMM_SMEM_BYTES = 1024 /* alignment slack */ + GEMM_STAGES * GEMM_STAGE_BYTES + 256 /* barriers */;
constexpr int GEMM_MAX_K_CHUNKS = 4;     // all-gather flags per 128-row block
// CTA-pair kernel (cta_group::2): per CTA and stage 128 rows of A and half of the 256-row B tile.
constexpr uint32_t GEMM_PAIR_STAGE_BYTES = GEMM_STAGE_A_BYTES + GEMM_STAGE_B_BYTES / 2;
constexpr int GEMM_PAIR_STAGES = 6;
constexpr int GEMM_TAIL_BOX = 32;        // rows of A per load of a tile that is computed as C^T (a row block that is not full)
constexpr uint32_t GEMM_TAIL_BOX_BYTES = GEMM_TAIL_BOX * GEMM_BK * 2;
constexpr size_t GEMM_PAIR_SMEM_BYTES = 1024 /* alignment slack */ + GEMM_PAIR_STAGES * GEMM_PAIR_STAGE_BYTES + 1024 /* barriers */ +
                                        GEMM_BM * 256 /* epilogue staging tile */;

enum GemmMode : int32_t {
    GEMM_PLAIN = 0,
    GEMM_ALL_GATHER = 1,      // A is gathered: local shard + staging filled by peers
    GEMM_REDUCE_SCATTER = 2,  // C is reduce-scattered: partial tiles pushed to the row owner
    GEMM_GROUPED = 3,         // rows of A grouped by expert, one weight per group, row counts read on the device
};
constexpr int GEMM_MAX_GROUPS = 64;      // groups of one launch (their row and tile offsets live in shared memory)

struct GemmArgs {
    CUtensorMap tmapA;        // A [M, K] row-major (all-gather: the staging buffer [R * shardRows, K])
    CUtensorMap tmapALocal;   // all-gather: this rank's shard [shardRows, K]
    CUtensorMap tmapB;        // B [N, K] row-major (the weight; C = A x B^T)
    CUtensorMap tmapTail;     // CTA-pair kernel, plain and grouped modes: A again, boxes of GEMM_TAIL_BOX rows
    uint8_t *c;               // plain / all-gather: C [M, N]; reduce-scatter: out [shardRows, N]
    const uint8_t *aLocal;    // all-gather: shard to push to the peers
    CommArgs *comm;
    int32_t *status;          // device int, set non-zero when a pipeline wait gave up
    int64_t magic;
    int32_t mode;
    int32_t M, N, K;          // M = rows of the whole product (R * shardRows in the fused modes)
    int32_t mBlocks, nBlocks, kBlocks;
    int32_t shardRows;        // rows per rank in the fused modes
    int32_t blocksPerShard;   // shardRows / GEMM_BM
    int32_t kChunks;          // all-gather: flags per row block
    int32_t flagStride;       // flags of one (source, destination) pair: the flag plane divided by the rank count
    int32_t kBlocksPerChunk;
    uint32_t commBlocks;      // all-gather: leading CTAs that push the local shard to the peers first
    uint32_t commTilesPerPair; // CTA-pair kernel: tiles (taken from the END of the walk) that each pushing pair computes afterwards
    uint32_t stageHandle;     // registry handle of the staging buffer (A staging or partial-C staging)
    uint64_t stageOffset;
    uint32_t isBf16;
    int32_t rasterGroup;      // CTA-pair kernel, plain mode: 256-row blocks per group of the tile walk
    // 8-bit operands (CTA-pair kernel, plain mode): 0 = 16-bit operands per isBf16, 1 = fp8 e4m3, 2 = fp8 e5m2.
    // A stage still holds one 128-byte swizzle row per operand row, i.e. 128 elements of K, and one tcgen05.mma
    // (kind::f8f6f4) covers 32 of them; C = alpha * A x B^T is written in the 16-bit type named by isBf16.
    int32_t fp8Format;
    float alpha;
    // Grouped mode (CTA-pair kernel): A [M, K] holds the rows of group 0, then group 1, ...; groupRows[g] of them (a
    // device array, so that no host round trip separates the kernel that counted the rows from this one).  B is
    // [groupsTotal * N, K], the weight of group g in rows [g * N, (g + 1) * N); C [M, N].  One launch covers groups
    // [groupBase, groupBase + groups).
    const int64_t *groupRows;
    int32_t groups, groupBase, groupsTotal;
    // Epilogue of the CTA-pair kernel (plain and grouped modes): 0 stores the product; 1 treats the columns as
    // (gate, up) pairs -- weight row 2i the gate row i, row 2i+1 the up row i -- and stores silu(gate) * up, so C is
    // [M, N / 2] and the [M, N] intermediate of a SwiGLU feed-forward never reaches memory.
    int32_t epilogue;
};
enum GemmEpilogue : int32_t { GEMM_EPI_STORE = 0, GEMM_EPI_SWIGLU = 1 };

// Block-scaled fp8 GEMM (gemm_tcgen05_fp8_block.cu): warp 0 TMA, warp 1 MMA, warps 4-11 fold the scratch accumulators.
constexpr unsigned GEMM_FP8_BLOCK_THREADS = 384;
constexpr int GEMM_FP8_BLOCK_STAGES = 5;     // one stage less than the bf16 kernel: scales and staging tiles live in shared memory too
constexpr int GEMM_FP8_SLICE_BOX = 16;       // rows of B per load of a slice
constexpr int GEMM_FP8_BLOCK_SCALE_SEG = 28; // most blocks of K whose scales are brought to shared memory at a time, twice: one in use, one on its way
constexpr uint32_t GEMM_FP8_BLOCK_SCALES_BYTES = GEMM_BM * (GEMM_FP8_BLOCK_SCALE_SEG + 1) * 4;
constexpr uint32_t GEMM_FP8_BLOCK_STAGE_C_BYTES = 8 * 32 * 128;      // eight promoter warps, 32 rows of 128 bytes each
constexpr size_t GEMM_FP8_BLOCK_SMEM_BYTES = 1024 /* alignment slack */ + GEMM_FP8_BLOCK_STAGES * GEMM_PAIR_STAGE_BYTES + 1024 /* barriers, weight scales */ +
                                             2 * GEMM_FP8_BLOCK_SCALES_BYTES + GEMM_FP8_BLOCK_STAGE_C_BYTES;

struct GemmBlockArgs {
    CUtensorMap tmapA;        // A [M, K] 8-bit, box 128 rows x 128 bytes
    CUtensorMap tmapALocal;   // all-gather: this rank's shard [shardRows, K]
    CUtensorMap tmapB;        // B [N, K] 8-bit, box 128 rows x 128 bytes
    CUtensorMap tmapBSlice;   // B again, box GEMM_FP8_SLICE_BOX rows x 128 bytes
    const float *scaleA;      // [M, K / 128]
    const float *scaleB;      // [scaleBRows, K / 128], one row per 128 rows of B
    uint8_t *c;               // [M, N] bf16 or fp16
    int32_t *status;
    int32_t M, N, K;
    int32_t nBlocks;          // 256-column tiles
    int32_t kBlocks;          // K / 128
    int32_t scaleBRows;       // ceil(N / 128)
    int32_t rasterGroup;
    // The first wideTiles tiles of the walk are computed whole (256 columns), the others in slices of sliceWidth columns (128, 64 or 32;
    // 256 where there are none): `items` pieces of work altogether.  PlanFp8Slices (gemm_few_rows.h)
    int32_t wideTiles, sliceWidth, items;
    uint32_t isBf16;
    int32_t fp8Format;        // 1 = e4m3, 2 = e5m2
    // Fused modes (GemmMode).  ALL_GATHER: tmapA and scaleA describe THIS rank's staging buffers ([R * shardRows, K] rows,
    // [R * shardRows, K / 128] scales, both registered on every rank); every rank writes its shard and the shard's
    // scales into all of them while the tiles are computed, and a tile of a peer's rows starts when the flag of its 128
    // rows is up (its own rows are read from the shard).
    // REDUCE_SCATTER: every 128 x 256 partial tile is stored into the row owner's partial staging buffer
    // ([R, shardRows, N] 16-bit, registered) and the owner adds the R partials in rank order into c [shardRows, N].
    int32_t mode;
    CommArgs *comm;
    int64_t magic;
    const uint8_t *aLocal;    // all-gather: [shardRows, K]
    const float *scaleALocal; // all-gather: [shardRows, K / 128]
    uint32_t aHandle, sHandle, outHandle;
    uint64_t aOffset, sOffset, outOffset;
    int32_t shardRows, blocksPerShard, flagStride;
};

// GEMM for few rows (gemm_tcgen05_skinny.cu): 128 rows of the weight x tn rows of A per tile, two CTAs per SM.
constexpr unsigned GEMM_SKINNY_THREADS = 192;
constexpr int GEMM_SKINNY_MAX_STAGES = 6;
constexpr uint32_t GEMM_SKINNY_W_BYTES = 128 * 128;
constexpr uint32_t GEMM_SKINNY_STATE_BYTES = 256;
constexpr uint32_t GEMM_SKINNY_RING_BYTES = 110592;      // stages x (16 KB + 128 tn): six of 18 KB down to three of 32 KB
constexpr size_t GEMM_SKINNY_SMEM_BYTES = 1024 /* alignment slack */ + GEMM_SKINNY_RING_BYTES + GEMM_SKINNY_STATE_BYTES +
                                          2 * (GEMM_SKINNY_MAX_GROUPS + 1) * 4;
static_assert(2 * (GEMM_SKINNY_SMEM_BYTES + 1024) <= 228 * 1024, "two CTAs share an SM");

struct SkinnyArgs {
    CUtensorMap tmapW;        // B [groupsTotal * N, K], box 128 rows x 64 columns
    CUtensorMap tmapX;        // A [M, K], box tn rows x 64 columns
    uint8_t *c;               // [M, N], or [M, N / 2] with the SwiGLU epilogue
    int32_t *status;
    const int64_t *groupRows; // grouped: rows per group on the device; null: one product
    int32_t M, N, K;
    int32_t kBlocks, nTiles;  // 64-wide steps of K, 128-column tiles of N
    int32_t tn, stages, split;
    int32_t groups, groupBase;
    uint32_t isBf16;
    int32_t epilogue;
};
const void *GemmSkinnyKernel();

#if defined(__CUDACC__)
// Where the rows and the row blocks (of `blockRows`) of groups groupBase .. groupBase + groups - 1 start, with the total behind
// the last group; a whole warp.  Counts below zero count as zero and rows past M do not exist.  The counts are fetched by 32
// lanes at a time: one lane after the other it was a chain of loads in front of every tile of the launch.
__device__ __forceinline__ void BuildGroupTable(const int64_t *groupRows, int groupBase, int groups, int M, int blockRows, int lane, int *rowStart,
                                                int *blockStart)
{
    long long before = 0;
    for (int g = lane; g < groupBase; g += 32) before += max(0ll, static_cast<long long>(groupRows[g]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    int blocks = 0;                                            // row blocks of the groups before this step's
    for (int base = 0; base < groups; base += 32) {
        const int g = base + lane;
        long long end = g < groups ? max(0ll, static_cast<long long>(groupRows[groupBase + g])) : 0ll;
        const long long own = end;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long up = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += up;
        }
        end += before;
        const int last = static_cast<int>(min(end, static_cast<long long>(M)));
        const int start = static_cast<int>(min(end - own, static_cast<long long>(M)));
        const int mine = (last - start + blockRows - 1) / blockRows;
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (g < groups) {
            rowStart[g] = start;
            blockStart[g] = blocks + incl - mine;
            if (g == groups - 1) {
                rowStart[groups] = last;
                blockStart[groups] = blocks + incl;
            }
        }
        before = __shfl_sync(0xffffffffu, end, 31);
        blocks += __shfl_sync(0xffffffffu, incl, 31);
    }
}
#endif

const void *StageCopyKernel();                       // (dst0, src0, vecs0, dst1, src1, vecs1), 256 threads a block
const void *GemmFp8BlockKernel(int mode);            // a kernel per GemmMode (plain, all-gather, reduce-scatter)
const void *GemmFp8BlockKernelEmulated(int mode);    // all-gather, reduce-scatter
const void *GemmKernelSingle();
const void *GemmKernelEmulated();
const void *GemmPairKernel();
const void *GemmPairKernelEmulated();

} // namespace TileXR

#endif
