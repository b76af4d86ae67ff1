// Router logits of a mixture-of-experts block: logits[T, E] = x[T, H] * gate[E, H]^T with 16-bit tokens, an fp32 gate and
// fp32 fused multiply-adds throughout.
//
// The library's fp32 product wants fp32 tokens (a copy of twice the size) and has no tile for a few dozen columns: 4096 x 7168
// by 32 experts took 83 us for the copy and 141 us for the product.  Here a block takes 64 tokens (32 where there are no more) x 32 experts; its eight
// warps share the K of a chunk, so that every lane owns, say, 8 x 8 results and reads 24 16-byte pieces of shared memory for 512
// multiply-adds (16 x 8 results per lane were no faster: 70 us where this takes 66); chunks of 256 elements arrive with
// cp.async two deep while the previous one is used.  K is split over the CTAs
// of a cluster until the chip is full; the partial tiles meet in distributed shared memory and are added in split order.
// Bound by the issue of the multiply-adds from a dozen experts on: 4096 x 7168 by 32 experts 66 us, by 256 experts 457 us, about
// 45 % of the fp32 peak.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cstdio>

#include <cuda_runtime_api.h>

#include "device/tilexr_platform.cuh"
#include "ep_kernels.cuh"
#include "tilexr_types.h"

namespace TileXR {

namespace {

constexpr int RL_EXPERTS = 32;
constexpr int RL_THREADS = 256;
constexpr int RL_WARP_K = 32;                                  // K of one warp per chunk
constexpr int RL_CHUNK = RL_WARP_K * RL_THREADS / 32;          // 256
constexpr int RL_X_PITCH = RL_CHUNK * 2 + 16;                  // bytes; an odd number of 16-byte units keeps the rows on different banks
constexpr int RL_G_PITCH = RL_CHUNK * 4 + 16;
constexpr int RL_MAX_SPLIT = 8;
constexpr int RlStageBytes(int tokens) { return tokens * RL_X_PITCH + RL_EXPERTS * RL_G_PITCH; }
constexpr int RlSmemBytes(int tokens) { return 2 * RlStageBytes(tokens); }
static_assert(RL_THREADS / 32 * 64 * RL_EXPERTS * 4 <= RlSmemBytes(64) && RL_THREADS / 32 * 32 * RL_EXPERTS * 4 <= RlSmemBytes(32),
              "the warps' tiles fit the stages");

struct RouterArgs {
    const uint8_t *x;
    const float *gate;
    float *out;
    int32_t T, H, E, split, bf16;
};

__device__ __forceinline__ void CpAsync16(uint32_t dst, const void *src, int bytes)
{
    // `bytes` (0 or 16) are read, the rest of the 16 is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <bool BF16>
__device__ __forceinline__ float2 Widen(uint32_t w)
{
    if (BF16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    return __half22float2(*reinterpret_cast<const __half2 *>(&w));
}

// Starts the copies of chunk `k0` (elements k0 .. k0 + 255, none past kEnd) into `stage`.
template <int RL_TOKENS>
__device__ __forceinline__ void LoadChunk(const RouterArgs &a, uint32_t stage, int t0, int e0, int k0, int kEnd, int tid)
{
    for (int i = tid; i < RL_TOKENS * (RL_CHUNK / 8); i += RL_THREADS) {
        const int r = i / (RL_CHUNK / 8), c = i % (RL_CHUNK / 8);
        const int k = k0 + c * 8;
        const bool in = t0 + r < a.T && k < kEnd;
        CpAsync16(stage + r * RL_X_PITCH + c * 16, in ? a.x + (static_cast<int64_t>(t0 + r) * a.H + k) * 2 : a.x, in ? 16 : 0);
    }
    const uint32_t g = stage + RL_TOKENS * RL_X_PITCH;
    for (int i = tid; i < RL_EXPERTS * (RL_CHUNK / 4); i += RL_THREADS) {
        const int r = i / (RL_CHUNK / 4), c = i % (RL_CHUNK / 4);
        const int k = k0 + c * 4;
        const bool in = e0 + r < a.E && k < kEnd;
        CpAsync16(g + r * RL_G_PITCH + c * 16, in ? a.gate + static_cast<int64_t>(e0 + r) * a.H + k : a.gate, in ? 16 : 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// I tokens and 8 experts per lane: a block takes 8 I tokens.
template <bool BF16, int I>
__global__ void __launch_bounds__(RL_THREADS, 1) RouterLogitsKernel(const RouterArgs a)
{
    constexpr int RL_TOKENS = 8 * I;
    constexpr int RL_STAGE_BYTES = RlStageBytes(RL_TOKENS);
    constexpr int RL_TILE = RL_TOKENS * RL_EXPERTS;
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t smemAddr = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = static_cast<int>(blockIdx.x) % a.split;               // clusters are `split` consecutive CTAs
    const int t0 = static_cast<int>(blockIdx.x) / a.split * RL_TOKENS;
    const int e0 = static_cast<int>(blockIdx.y) * RL_EXPERTS;
    // the parts of K are whole chunks; a part may be empty, its tile is zero
    const int chunksAll = (a.H + RL_CHUNK - 1) / RL_CHUNK;
    const int per = (chunksAll + a.split - 1) / a.split;
    const int kBegin = min(a.H, part * per * RL_CHUNK);
    const int kEnd = min(a.H, kBegin + per * RL_CHUNK);
    const int chunks = (kEnd - kBegin + RL_CHUNK - 1) / RL_CHUNK;

    // lane: tokens i * 8 + tg, experts j * 4 + eg
    const int tg = lane >> 2, eg = lane & 3;
    float acc[I][8];
#pragma unroll
    for (int i = 0; i < I; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    }
    tilexr::StreamRelease();
    tilexr::StreamWait();
    if (chunks > 0) LoadChunk<RL_TOKENS>(a, smemAddr, t0, e0, kBegin, kEnd, tid);
    for (int c = 0; c < chunks; ++c) {
        if (c + 1 < chunks) {
            LoadChunk<RL_TOKENS>(a, smemAddr + ((c + 1) & 1) * RL_STAGE_BYTES, t0, e0, kBegin + (c + 1) * RL_CHUNK, kEnd, tid);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint8_t *xs = smem + (c & 1) * RL_STAGE_BYTES + warp * RL_WARP_K * 2;
        const uint8_t *gs = smem + (c & 1) * RL_STAGE_BYTES + RL_TOKENS * RL_X_PITCH + warp * RL_WARP_K * 4;
#pragma unroll 1
        for (int k = 0; k < RL_WARP_K; k += 8) {
            float4 gv[2][8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                gv[0][j] = *reinterpret_cast<const float4 *>(gs + (j * 4 + eg) * RL_G_PITCH + k * 4);
                gv[1][j] = *reinterpret_cast<const float4 *>(gs + (j * 4 + eg) * RL_G_PITCH + k * 4 + 16);
            }
#pragma unroll
            for (int i = 0; i < I; ++i) {
                const uint4 xv = *reinterpret_cast<const uint4 *>(xs + (i * 8 + tg) * RL_X_PITCH + k * 2);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float2 lo = Widen<BF16>(half == 0 ? xv.x : xv.z);
                    const float2 hi = Widen<BF16>(half == 0 ? xv.y : xv.w);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(lo.x, gv[half][j].x, acc[i][j]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(lo.y, gv[half][j].y, acc[i][j]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(hi.x, gv[half][j].z, acc[i][j]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(hi.y, gv[half][j].w, acc[i][j]);
                }
            }
        }
        __syncthreads();                                       // the stage may be filled again
    }
    // the warps' tiles, then the block's tile in the first of them
    float *tiles = reinterpret_cast<float *>(smem);
#pragma unroll
    for (int i = 0; i < I; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) tiles[warp * RL_TILE + (i * 8 + tg) * RL_EXPERTS + j * 4 + eg] = acc[i][j];
    }
    __syncthreads();
    for (int o = tid; o < RL_TILE; o += RL_THREADS) {
        float v = tiles[o];
#pragma unroll
        for (int w = 1; w < RL_THREADS / 32; ++w) v += tiles[w * RL_TILE + o];
        tiles[o] = v;
    }
    if (a.split > 1) {
        __syncthreads();
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    const int rows = RL_TOKENS / a.split;
    for (int o = tid; o < rows * RL_EXPERTS; o += RL_THREADS) {
        const int at = part * rows * RL_EXPERTS + o;
        float v = 0.f;
        if (a.split == 1) {
            v = tiles[at];
        } else {
            for (int s = 0; s < a.split; ++s) {
                uint32_t remote;
                float u;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smemAddr + at * 4), "r"(s));
                asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(u) : "r"(remote) : "memory");
                v = s == 0 ? u : v + u;
            }
        }
        const int t = t0 + at / RL_EXPERTS, e = e0 + at % RL_EXPERTS;
        if (t < a.T && e < a.E) a.out[static_cast<int64_t>(t) * a.E + e] = v;
    }
    if (a.split > 1) {
        // nobody leaves while its tile may still be read
        __syncthreads();
        asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

} // namespace

template <bool BF16, int I>
static const void *RouterKernel() { return reinterpret_cast<const void *>(&RouterLogitsKernel<BF16, I>); }

int LaunchRouterLogits(const void *x, const float *gate, int64_t tokens, int64_t h, int64_t experts, bool bf16, float *out, void *stream)
{
    // Few tokens: a smaller tile, so that no block computes rows that do not exist (32 x 2048 by 64 experts: 12.1 -> 8.7 us).
    const int perBlock = tokens <= 32 ? 32 : 64;
    const void *kernel = perBlock == 32 ? (bf16 ? RouterKernel<true, 4>() : RouterKernel<false, 4>()) : (bf16 ? RouterKernel<true, 8>() : RouterKernel<false, 8>());
    const int64_t tokenTiles = (tokens + perBlock - 1) / perBlock;
    RouterArgs a{static_cast<const uint8_t *>(x), gate, out, static_cast<int32_t>(tokens), static_cast<int32_t>(h), static_cast<int32_t>(experts), 1,
                 bf16 ? 1 : 0};
    const int64_t tiles = tokenTiles * ((experts + RL_EXPERTS - 1) / RL_EXPERTS);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // one block per SM: K is split while the parts still fit beside one another and hold a chunk each
    while (a.split < RL_MAX_SPLIT && tiles * a.split * 2 <= sms && a.split * 2 * RL_CHUNK <= h + RL_CHUNK - 1) a.split *= 2;
    void *params[] = {&a};
    // the limit belongs to the kernel on the current device: raised on every call, so that a second device of the process has it, too
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RlSmemBytes(perBlock));
    if (e == cudaSuccess) {
        e = static_cast<cudaError_t>(LaunchOverlapped(kernel, static_cast<unsigned>(tokenTiles * a.split), static_cast<unsigned>((experts + RL_EXPERTS - 1) / RL_EXPERTS),
                                                      RL_THREADS, static_cast<size_t>(RlSmemBytes(perBlock)), static_cast<unsigned>(a.split), params, stream));
    }
    if (e != cudaSuccess) {
        fprintf(stderr, "[TileXR] router logits launch failed: %s\n", cudaGetErrorString(e));
        cudaGetLastError();
        return TILEXR_ERROR_RUNTIME;
    }
    NoteLaunch();
    return TILEXR_SUCCESS;
}

} // namespace TileXR
