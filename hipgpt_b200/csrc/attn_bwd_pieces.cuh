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

// The same of an operand as three bf16 pieces; the six products of such pieces that count, small ones first
template <int D>
constexpr int kBlock3 = 3 * Img<D>::kPiece;
template <int D>
constexpr int kTileBytes3 = (kTile / 8) * kBlock3<D>;
__device__ constexpr int kExactA[6] = {0, 2, 1, 0, 1, 0}, kExactB[6] = {2, 0, 1, 1, 0, 0};

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

// Two fp32 numbers -> three words of two bf16 each whose sums are the numbers (to 2^-25 of them, whatever their magnitude)
__device__ __forceinline__ void cut3(float2 x, uint32_t &h, uint32_t &m, uint32_t &l)
{
    h = pack_bf16(x.x, x.y);
    const float2 r = fadd2(x, make_float2(-__uint_as_float(h << 16), -__uint_as_float(h & 0xffff0000u)));
    m = pack_bf16(r.x, r.y);
    const float2 s = fadd2(r, make_float2(-__uint_as_float(m << 16), -__uint_as_float(m & 0xffff0000u)));
    l = pack_bf16(s.x, s.y);
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
