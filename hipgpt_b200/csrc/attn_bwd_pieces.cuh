// What the kernels of the attention backward on the tensor pipe share: operands as two fp16 pieces, and their images.
#pragma once

#include "tc_primitives.cuh"

#include <cuda_fp16.h>

namespace hipgpt {
namespace {

constexpr int kLanes = 128;            // rows (or keys) per block = TMEM lanes
constexpr int kTile = 64;              // columns per tile

// Sizes of an operand image, in bytes.
template <int D>
struct Img {
    static constexpr int kPiece = (D / 8) * 128;     // one piece of an 8-row block
    static constexpr int kBlock = 2 * kPiece;        // an 8-row block
    static constexpr int kTileBytes = (kTile / 8) * kBlock;     // 64 rows
};

// Two fp32 numbers below 2^16 -> two words of two fp16 each whose sums are the numbers (to 2^-23 of them, 2^-25 where that is more).
// An infinity leaves a NaN.
__device__ __forceinline__ void cut2(float2 x, uint32_t &h, uint32_t &l)
{
    const __half2 hh = __float22half2_rn(x);
    const float2 back = __half22float2(hh);
    const __half2 ll = __float22half2_rn(ffma2(back, make_float2(-1.0f, -1.0f), x));
    h = *reinterpret_cast<const uint32_t *>(&hh);
    l = *reinterpret_cast<const uint32_t *>(&ll);
}

// The power of two that brings a largest magnitude into [2^14, 2^15), and one over it, from the magnitude's bits.  Magnitudes
// below 2^-100 are treated as that; an infinite one leaves both normal numbers.
__device__ __forceinline__ uint32_t range_exponent(uint32_t bits) { return max(bits & 0x7f800000u, 27u << 23); }
__device__ __forceinline__ float range_up(uint32_t e) { return __uint_as_float((268u << 23) - e); }
__device__ __forceinline__ float range_down(uint32_t e) { return __uint_as_float(e - (14u << 23)); }

}  // namespace
}  // namespace hipgpt
