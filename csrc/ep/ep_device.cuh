// Device code that the expert-parallel kernels share: routing of a token, ranking of a block's routes, quantisation of rows.
#ifndef TILEXR_EP_DEVICE_CUH
#define TILEXR_EP_DEVICE_CUH

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "device/tilexr_convert.cuh"
#include "device/tilexr_rma.cuh"
#include "device/tilexr_sync.cuh"
#include "ep_kernels.cuh"
#include "tilexr_ep.h"

namespace TileXR {

using namespace tilexr;

namespace {

// One kernel per kind of transport: with all of them in one the registers of a 512-thread block (64, two blocks per SM) ran
// out (628 bytes of spill loads against 340; 4096 x 7168 fp8 96 -> 92 us).
enum EpTransport : int { EP_PLAIN = 0, EP_FP8 = 1, EP_MXFP8 = 2, EP_INT8 = 3, EP_FP8_ROUND = 4 };   // the last: fp8 and back, one rank only

constexpr float FP8_E4M3_MAX = 448.0f;
constexpr float FP8_AMAX_FLOOR = 1e-4f;

__device__ __forceinline__ float WarpMax(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float WarpSum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ uint32_t Fp8x4(float a, float b, float c, float d)
{
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
    return lo | (hi << 16);
}

__device__ __forceinline__ uint32_t Fp8x4E5m2(float a, float b, float c, float d)
{
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E5M2);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E5M2);
    return lo | (hi << 16);
}

// ---- routing: one warp scores one token and picks its top-k -------------------------------------------
// Lane l owns experts l, l+32, ...  Selection is by score (+ optional bias), ties go to the
// lower expert id; the gate weight is the unbiased score, optionally renormalised over the
// selected experts and multiplied by `routedScale`.
template <int PER_LANE>
__device__ __forceinline__ int RouteTokenN(const float *logits, const float *bias, int numExperts, int topK, int scoreFunc,
                                            int renormalize, float routedScale, int lane, int32_t *idsOut, float *weightsOut, float *picked)
{
    float score[PER_LANE];
    float sel[PER_LANE];
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const int e = j * 32 + lane;
        score[j] = e < numExperts ? logits[e] : -INFINITY;
        mx = fmaxf(mx, score[j]);
    }
    if (scoreFunc == TileXREp::TILEXR_EP_SCORE_SOFTMAX) {
        mx = WarpMax(mx);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) {
            const int e = j * 32 + lane;
            score[j] = e < numExperts ? expf(score[j] - mx) : 0.f;
            sum += score[j];
        }
        sum = WarpSum(sum);
        const float inv = 1.0f / sum;
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) score[j] *= inv;
    } else {
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) {
            const int e = j * 32 + lane;
            score[j] = e < numExperts ? 1.0f / (1.0f + expf(-score[j])) : 0.f;
        }
    }
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
        const int e = j * 32 + lane;
        sel[j] = e < numExperts ? score[j] + (bias != nullptr ? bias[e] : 0.f) : -INFINITY;
    }
    float myWeight = 0.f;   // lane k keeps the k-th pick
    int myId = -1;
    float total = 0.f;
    for (int k = 0; k < topK; ++k) {
        float best = -INFINITY;
        int bestE = 0x7fffffff;
        float bestScore = 0.f;
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) {
            const int e = j * 32 + lane;
            if (sel[j] > best) {   // ascending e within a lane: first maximum wins the tie
                best = sel[j];
                bestE = e;
                bestScore = score[j];
            }
        }
        // The lanes' maxima are compared as integers of the same order (a zero of either sign is one value; a lane without
        // a candidate, whose scores are NaN, minus infinity or used up, has the smallest key): two warp reductions and a
        // shuffle per pick instead of fifteen shuffles.
        const uint32_t bits = __float_as_uint(best + 0.f);
        const uint32_t key = bestE == 0x7fffffff ? 0u : (bits & 0x80000000u) != 0 ? ~bits : bits | 0x80000000u;
        const uint32_t top = __reduce_max_sync(0xffffffffu, key);
        bestE = static_cast<int>(__reduce_min_sync(0xffffffffu, key == top ? static_cast<uint32_t>(bestE) : 0x7fffffffu));
        bestScore = __shfl_sync(0xffffffffu, bestScore, bestE & 31);
        if (top == 0u) bestScore = 0.f;
        if ((bestE & 31) == lane) {
#pragma unroll
            for (int j = 0; j < PER_LANE; ++j) {
                if (j == (bestE >> 5)) sel[j] = -INFINITY;
            }
        }
        if (lane == k) {
            myWeight = bestScore;
            myId = bestE;
        }
        total += bestScore;
    }
    if (lane < topK) {
        float w = myWeight;
        if (renormalize) w = w / total;
        w *= routedScale;
        idsOut[lane] = myId;
        weightsOut[lane] = w;
        *picked = w;
    }
    return myId;
}

// The per-lane score table is sized for the expert count, so that 256 experts keep 8 scores per lane in
// registers instead of the 32 that the largest supported count needs.  Returns the expert that lane k picked k-th, and its gate
// weight in *picked.
__device__ __forceinline__ int RouteToken(const float *logits, const float *bias, int numExperts, int topK, int scoreFunc,
                                           int renormalize, float routedScale, int lane, int32_t *idsOut, float *weightsOut, float *picked)
{
    if (numExperts <= 256) {
        return RouteTokenN<8>(logits, bias, numExperts, topK, scoreFunc, renormalize, routedScale, lane, idsOut, weightsOut, picked);
    }
    if (numExperts <= 512) {
        return RouteTokenN<16>(logits, bias, numExperts, topK, scoreFunc, renormalize, routedScale, lane, idsOut, weightsOut, picked);
    }
    return RouteTokenN<EP_MAX_EXPERTS / 32>(logits, bias, numExperts, topK, scoreFunc, renormalize, routedScale, lane, idsOut, weightsOut, picked);
}

// What KernelEpilogue keeps but for the status, by one thread and without waiting for the other blocks.
__device__ __forceinline__ void EndLocalLaunch(CommArgs *c, const Waiter &w)
{
    c->dfx[TILEXR_DFX_LAUNCHES] += 1;
    st_relaxed_sys_u64(CtrlWord(c, c->rank, TILEXR_CTRL_DONE_WORD + c->rank), MakeFlag(w.epoch, 0));
    *CtrlWord(c, c->rank, TILEXR_CTRL_EPOCH_WORD) = w.epoch;
}

__device__ __forceinline__ void Fp8Unpack8(uint2 raw, __nv_fp8_interpretation_t kind, float s, float *f)
{
    const uint32_t w[2] = {raw.x, raw.y};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const __half2_raw h2 = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>((w[i] >> (16 * j)) & 0xffffu), kind);
            const float2 f2 = __half22float2(*reinterpret_cast<const __half2 *>(&h2));
            f[i * 4 + j * 2] = f2.x * s;
            f[i * 4 + j * 2 + 1] = f2.y * s;
        }
    }
}

// Sixteen elements per lane, eight neighbouring lanes share a block of 128: e4m3 values, and in *scales the four fp32 scales of the
// warp's 512 elements (16 bytes of the row's scales), the same in all lanes; the lane's own in *own.  Called by a whole warp.
__device__ __forceinline__ Vec16 QuantFp8Block16(const float *f, Vec16 *scales, float *own = nullptr)
{
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    amax = fmaxf(amax, FP8_AMAX_FLOOR);
    const float inv = FP8_E4M3_MAX / amax;
    const float scale = amax / FP8_E4M3_MAX;
    if (own != nullptr) *own = scale;
    scales->x = __float_as_uint(__shfl_sync(0xffffffffu, scale, 0));
    scales->y = __float_as_uint(__shfl_sync(0xffffffffu, scale, 8));
    scales->z = __float_as_uint(__shfl_sync(0xffffffffu, scale, 16));
    scales->w = __float_as_uint(__shfl_sync(0xffffffffu, scale, 24));
    Vec16 q;
    q.x = Fp8x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
    q.y = Fp8x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
    q.z = Fp8x4(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
    q.w = Fp8x4(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
    return q;
}

// MXFP8: 32 elements = 2 lanes share the exponent 2^(floor(log2 amax) - emax); *scales are the warp's 16 exponent bytes.
__device__ __forceinline__ Vec16 QuantMx16(const float *f, bool e5m2, int lane, Vec16 *scales)
{
    float amax = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(f[j]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    const int emax = e5m2 ? 15 : 8;
    int ex = -127;
    if (amax > 0.f) {
        const uint32_t biased = (__float_as_uint(amax) >> 23) & 0xffu;
        ex = (biased == 0 ? -126 : static_cast<int>(biased) - 127) - emax;
    }
    ex = max(-127, min(127, ex));
    const float inv = exp2f(static_cast<float>(-ex));
    uint32_t word = (lane & 1) == 0 ? static_cast<uint32_t>(ex + 127) << (8 * ((lane >> 1) & 3)) : 0u;
    word |= __shfl_xor_sync(0xffffffffu, word, 2);
    word |= __shfl_xor_sync(0xffffffffu, word, 4);
    scales->x = __shfl_sync(0xffffffffu, word, 0);
    scales->y = __shfl_sync(0xffffffffu, word, 8);
    scales->z = __shfl_sync(0xffffffffu, word, 16);
    scales->w = __shfl_sync(0xffffffffu, word, 24);
    Vec16 q;
    if (e5m2) {
        q.x = Fp8x4E5m2(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
        q.y = Fp8x4E5m2(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
        q.z = Fp8x4E5m2(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
        q.w = Fp8x4E5m2(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
    } else {
        q.x = Fp8x4(f[0] * inv, f[1] * inv, f[2] * inv, f[3] * inv);
        q.y = Fp8x4(f[4] * inv, f[5] * inv, f[6] * inv, f[7] * inv);
        q.z = Fp8x4(f[8] * inv, f[9] * inv, f[10] * inv, f[11] * inv);
        q.w = Fp8x4(f[12] * inv, f[13] * inv, f[14] * inv, f[15] * inv);
    }
    return q;
}

// Rank of each of a block's routes among its routes to the same column (expert[] -1: none), in (token, k) order, and the routes per column in hist[],
// which is zero before: one warp walks the routes 32 at a time; lanes with the same column find one another with a match and the last
// of them moves the column's running count on.
__device__ __forceinline__ void RankBlockRoutes(int routes, const int32_t *expert, int32_t *rank, int32_t *hist, int lane)
{
    for (int base = 0; base < routes; base += 32) {
        const int i = base + lane;
        const int e = i < routes ? expert[i] : -1;
        const uint32_t same = __match_any_sync(0xffffffffu, e);
        int r = 0;
        if (e >= 0) r = hist[e] + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (e >= 0 && (same & ~((2u << lane) - 1u)) == 0) hist[e] += __popc(same);
        __syncwarp();
        if (i < routes) rank[i] = r;
    }
}

// int8 rows with optional per-expert smoothing scales `sc` (null: none): the largest magnitude of a row of `chunks` 16-element pieces, the same in all
// lanes, and every `parts`-th 512 elements of it from `part` on, times `inv`, rounded and clamped.  Called by a whole warp.
__device__ __forceinline__ float Int8RowAmax(const uint8_t *row, const float *sc, int chunks, bool bf16, int lane)
{
    float amax = 0.f;
    for (int c = lane; c < chunks; c += 32) {
        float f[16];
        Unpack8(ld_vec16(row + static_cast<int64_t>(c) * 32), bf16, f);
        Unpack8(ld_vec16(row + static_cast<int64_t>(c) * 32 + 16), bf16, f + 8);
#pragma unroll
        for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(sc != nullptr ? f[j] * sc[c * 16 + j] : f[j]));
    }
    return WarpMax(amax);
}

__device__ __forceinline__ void Int8RowStore(const uint8_t *row, const float *sc, float inv, int chunks, bool bf16, int part, int parts, int lane, uint8_t *to)
{
    for (int c = part * 32 + lane; c < chunks; c += parts * 32) {
        float f[16];
        Unpack8(ld_vec16(row + static_cast<int64_t>(c) * 32), bf16, f);
        Unpack8(ld_vec16(row + static_cast<int64_t>(c) * 32 + 16), bf16, f + 8);
        uint32_t wds[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float v = (sc != nullptr ? f[j] * sc[c * 16 + j] : f[j]) * inv;
            const int q = max(-128, min(127, __float2int_rn(v)));
            wds[j >> 2] |= static_cast<uint32_t>(q & 0xff) << (8 * (j & 3));
        }
        st_vec16(to + static_cast<int64_t>(c) * 16, Vec16{wds[0], wds[1], wds[2], wds[3]});
    }
}

} // namespace

} // namespace TileXR

#endif
