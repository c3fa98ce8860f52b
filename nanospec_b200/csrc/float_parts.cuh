// A float times 2^24 as the sum of three bfloat16, each the rest of the one before rounded to nearest (8 + 8 + 8 bits).  Times 2^24 the last bit of
// every float, the smallest ones' 2^-149 too, lies above bfloat16's smallest normal number, so that the sum is exact for all below 2^104; from there
// on, and for an infinity or a NaN, a part is infinite and the next a NaN.  A product of two floats, 2^48 times too large, is kept as the six products
// of parts that reach 2^-24 of it; the two largest that are left out reach 2^-25 each.  Whoever adds such products looks at sums that are not
// finite (operands from 2^104 or products from 2^80 on do that too) and forms those from the floats.
#pragma once

#include "common.cuh"

namespace {

constexpr int kParts = 3;
constexpr float kPartsScale = 16777216.f;               // 2^24
constexpr float kPartsBack = 3.552713678800501e-15f;    // 2^-48, of a product

// a pair of floats as three pairs of bfloat16 (the first number in the low half)
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const float2 minus = make_float2(-1.f, -1.f), v = __fmul2_rn(make_float2(a, b), make_float2(kPartsScale, kPartsScale));
    __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    hi = *reinterpret_cast<uint32_t*>(&h);
    const float2 r = __ffma2_rn(make_float2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), minus, v);
    __nv_bfloat162 m = __floats2bfloat162_rn(r.x, r.y);
    mid = *reinterpret_cast<uint32_t*>(&m);
    const float2 q = __ffma2_rn(make_float2(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u)), minus, r);
    __nv_bfloat162 l = __floats2bfloat162_rn(q.x, q.y);
    lo = *reinterpret_cast<uint32_t*>(&l);
}

}  // namespace
