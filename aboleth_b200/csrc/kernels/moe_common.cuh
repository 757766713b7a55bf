// Device helpers shared by the MoE kernels: router softmax/top-k in one warp,
// 1 x group block-scaled e4m3 quantisation, and the record geometry.
//
// Record layout (one record per (token, destination rank); reference:
// python/aboleth/moe/compiled_plan.py:101-107, python/aboleth/moe/kernels.py:98-143):
//   payload row  : hidden x {bf16 | e4m3}
//   metadata row : int32 [token, n_selected, expert_id x k, weight_bits x k, scale_bits x cols]
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "common.cuh"

namespace ab::moe {

constexpr int kMaxTopK = 16;
constexpr int kMaxWorld = 32;
constexpr int kMaxExpertsPerLane = 16;  // experts <= 512
constexpr float kFp8Max = 448.0f;

__device__ __forceinline__ float bf16_lo(std::uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(std::uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

__device__ __forceinline__ std::uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<std::uint32_t *>(&v);
}

// scale = max(amax, floor) / 448, optionally rounded UP to a power of two.
__device__ __forceinline__ float quant_scale(float amax, float floor_, int round_pow2) {
    float scale = fmaxf(amax, floor_) / kFp8Max;
    if (round_pow2) {
        std::uint32_t bits = __float_as_uint(scale);
        if (bits & 0x007fffffu)
            bits = (bits & 0xff800000u) + 0x00800000u;
        scale = __uint_as_float(bits);
    }
    return scale;
}

// x / scale.  The default is the hardware's approximate division (about 2 ulp,
// far below an e4m3 quantum; a value that sits on a rounding tie may land on
// the other neighbour than IEEE division would pick).  Define
// ABOLETH_EXACT_QUANT_DIV for bit-exact IEEE division at several times the cost.
__device__ __forceinline__ float quant_div(float x, float scale) {
#ifdef ABOLETH_EXACT_QUANT_DIV
    return x / scale;
#else
    return __fdividef(x, scale);
#endif
}

// Four values times the reciprocal scale `inv` -> four e4m3 codes.  The conversion saturates at
// +-448 by itself, so no clamp is spent here (a NaN input stays NaN).
__device__ __forceinline__ std::uint32_t fp8x4(float a, float b, float c, float d, float inv) {
#ifdef ABOLETH_EXACT_QUANT_DIV
    const float scale = inv;  // the caller passes the scale itself
    a = quant_div(a, scale); b = quant_div(b, scale); c = quant_div(c, scale); d = quant_div(d, scale);
#else
    a *= inv; b *= inv; c *= inv; d *= inv;
#endif
    const std::uint32_t p0 = __nv_cvt_float2_to_fp8x2(make_float2(a, b), __NV_SATFINITE, __NV_E4M3);
    const std::uint32_t p1 = __nv_cvt_float2_to_fp8x2(make_float2(c, d), __NV_SATFINITE, __NV_E4M3);
    return p0 | (p1 << 16);
}

// The same for an `inv` that is a power of two, where multiplying and dividing agree.
__device__ __forceinline__ std::uint32_t fp8x4_scaled(float a, float b, float c, float d, float inv) {
    const std::uint32_t p0 = __nv_cvt_float2_to_fp8x2(make_float2(a * inv, b * inv), __NV_SATFINITE, __NV_E4M3);
    const std::uint32_t p1 = __nv_cvt_float2_to_fp8x2(make_float2(c * inv, d * inv), __NV_SATFINITE, __NV_E4M3);
    return p0 | (p1 << 16);
}

// Sixteen bf16 values (two 16-byte vectors) -> absolute maximum.  Signs are masked off two values
// at a time and the packed maximum unit compares them; one conversion at the end.
__device__ __forceinline__ float amax16(const uint4 &a, const uint4 &b) {
    const std::uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    __nv_bfloat162 m;
    *reinterpret_cast<std::uint32_t *>(&m) = w[0] & 0x7fff7fffu;
#pragma unroll
    for (int i = 1; i < 8; ++i) {
        __nv_bfloat162 v;
        *reinterpret_cast<std::uint32_t *>(&v) = w[i] & 0x7fff7fffu;
        m = __hmax2(m, v);
    }
    const std::uint32_t bits = *reinterpret_cast<std::uint32_t *>(&m);
    return fmaxf(bf16_lo(bits), bf16_hi(bits));
}

// Sixteen bf16 values -> sixteen e4m3 codes at `scale`.  The default multiplies by the correctly
// rounded reciprocal of the scale (exact for power-of-two scales, within 1.5 ulp of the division
// otherwise: far below an e4m3 quantum, so only a value that sits on a rounding tie can land on the
// other neighbouring code).  ABOLETH_EXACT_QUANT_DIV divides instead.
__device__ __forceinline__ uint4 quant16(const uint4 &a, const uint4 &b, float scale) {
#ifdef ABOLETH_EXACT_QUANT_DIV
    const float inv = scale;
#else
    const float inv = __frcp_rn(scale);
#endif
    uint4 q;
    q.x = fp8x4(bf16_lo(a.x), bf16_hi(a.x), bf16_lo(a.y), bf16_hi(a.y), inv);
    q.y = fp8x4(bf16_lo(a.z), bf16_hi(a.z), bf16_lo(a.w), bf16_hi(a.w), inv);
    q.z = fp8x4(bf16_lo(b.x), bf16_hi(b.x), bf16_lo(b.y), bf16_hi(b.y), inv);
    q.w = fp8x4(bf16_lo(b.z), bf16_hi(b.z), bf16_lo(b.w), bf16_hi(b.w), inv);
    return q;
}

// Reduce a maximum over the `width` consecutive lanes (power of two <= 32)
// that share one quantisation group.
__device__ __forceinline__ float group_max(float v, int width) {
    for (int off = width >> 1; off > 0; off >>= 1)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    return v;
}

__device__ __forceinline__ float logit_of(float v) { return v; }
__device__ __forceinline__ float logit_of(__nv_bfloat16 v) { return __bfloat162float(v); }

// One warp: softmax over `experts` logits and the `top_k` largest, ties to
// the lower index.  Lane l holds experts l, l+32, ...  On return lane j < top_k
// holds (id, weight) of the j-th choice.  `renormalize` divides the selected
// probabilities by their sum.
//
// A round is latency, not work, so it is kept short: values are order-preserving integer keys (0: nothing to
// choose - a NaN, minus infinity, or taken), a lane's largest key comes from a tree of integer maxima, and the
// lowest index that holds the warp's largest key from a second one; weights are computed once, after the rounds.
// (Floating-point compares in a chain, and a weight per round, made routing most of a decode-size dispatch.)
template <int PER_LANE, typename Logit>
__device__ __forceinline__ void warp_softmax_topk_n(const Logit *logits, int experts, int top_k,
                                                    int renormalize, int &out_id, float &out_w) {
    const int lane = threadIdx.x & 31;
    float v[PER_LANE];
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        const int e = lane + 32 * i;
        v[i] = e < experts ? logit_of(logits[e]) : -INFINITY;
        mx = fmaxf(mx, v[i]);
    }
    for (int off = 16; off > 0; off >>= 1)
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    float sum = 0.f;
    std::uint32_t key[PER_LANE];
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
        sum += (lane + 32 * i) < experts ? __expf(v[i] - mx) : 0.f;
        const std::uint32_t raw = __float_as_uint(v[i] + 0.0f);  // -0 becomes 0: equal logits have equal keys
        key[i] = v[i] > -INFINITY ? raw ^ ((raw >> 31) ? 0xffffffffu : 0x80000000u) : 0u;
    }
    for (int off = 16; off > 0; off >>= 1)
        sum += __shfl_xor_sync(0xffffffffu, sum, off);

    out_id = -1;
    std::uint32_t mine = 0;
    for (int j = 0; j < top_k; ++j) {
        std::uint32_t best = key[0];
#pragma unroll
        for (int i = 1; i < PER_LANE; ++i)
            best = max(best, key[i]);
        const std::uint32_t top = __reduce_max_sync(0xffffffffu, best);
        unsigned at = 0x7fffffffu;  // also what a round without a choice reports
#pragma unroll
        for (int i = PER_LANE - 1; i >= 0; --i)
            at = key[i] == top && top != 0 ? static_cast<unsigned>(lane + 32 * i) : at;
        const unsigned winner = __reduce_min_sync(0xffffffffu, at);
#pragma unroll
        for (int i = 0; i < PER_LANE; ++i)
            key[i] = static_cast<unsigned>(lane + 32 * i) == winner ? 0u : key[i];
        if (lane == j) {
            out_id = static_cast<int>(winner);
            mine = top;
        }
    }
    out_w = 0.f;
    if (lane < top_k) {
        const float value = mine == 0 ? -INFINITY
                                      : __uint_as_float(mine ^ ((mine >> 31) ? 0x80000000u : 0xffffffffu));
        out_w = __expf(value - mx) / sum;
    }
    if (renormalize) {
        float picked_sum = 0.f;
        for (int j = 0; j < top_k; ++j)
            picked_sum += __shfl_sync(0xffffffffu, out_w, j);
        if (picked_sum > 0.f)
            out_w /= picked_sum;
    }
}

template <typename Logit>
__device__ __forceinline__ void warp_softmax_topk(const Logit *logits, int experts, int top_k,
                                                  int renormalize, int &out_id, float &out_w) {
    if (experts <= 32)
        warp_softmax_topk_n<1>(logits, experts, top_k, renormalize, out_id, out_w);
    else if (experts <= 128)
        warp_softmax_topk_n<4>(logits, experts, top_k, renormalize, out_id, out_w);
    else if (experts <= 256)
        warp_softmax_topk_n<8>(logits, experts, top_k, renormalize, out_id, out_w);
    else
        warp_softmax_topk_n<kMaxExpertsPerLane>(logits, experts, top_k, renormalize, out_id, out_w);
}

}  // namespace ab::moe
