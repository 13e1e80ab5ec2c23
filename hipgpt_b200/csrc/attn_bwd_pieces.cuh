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

// Two fp32 numbers up to 2^15 -> two words of two fp16 each, hi and 2^12 times what hi leaves: hi + 2^-12 lo is the number to 2^-23 of it
// down to 2^-14, to 2^-37 below.  (Without the factor the low piece ran into fp16's smallest numbers at 2^-2 already.)  The products with one low piece are 2^12
// times too large then, that of two 2^24: the tensor core brings the accumulator down where the next larger products start.
// An infinity leaves a NaN.
constexpr int kLowShift = 12;
constexpr float kLowUp = 4096.0f, kLowDown = 1.0f / 4096.0f;
__device__ __forceinline__ void cut2(float2 x, uint32_t &h, uint32_t &l)
{
    const __half2 hh = __float22half2_rn(x);
    const float2 back = __half22float2(hh);
    const __half2 ll = __float22half2_rn(fmul2(ffma2(back, make_float2(-1.0f, -1.0f), x), make_float2(kLowUp, kLowUp)));
    h = *reinterpret_cast<const uint32_t *>(&hh);
    l = *reinterpret_cast<const uint32_t *>(&ll);
}

// The power of two that brings a largest magnitude into [2^14, 2^15), and one over it, from the magnitude's bits.  Magnitudes
// below 2^-100 are treated as that; an infinite one leaves both normal numbers.
__device__ __forceinline__ uint32_t range_exponent(uint32_t bits) { return max(bits & 0x7f800000u, 27u << 23); }
__device__ __forceinline__ float range_up(uint32_t e) { return __uint_as_float((268u << 23) - e); }
__device__ __forceinline__ float range_down(uint32_t e) { return __uint_as_float(e - (14u << 23)); }
// The most that two such factors make together: not infinite, so that a row of zeros stays one beside rows whose scores leave fp32
constexpr float kFacMost = 1e38f;

}  // namespace
}  // namespace hipgpt
