// A float as the sum of three bfloat16, each the rest of the one before rounded to nearest (8 + 8 + 8 bits: exact but for numbers near
// the ends of the exponent's range; parts of an infinity or a NaN make a NaN).  A product of two floats is kept as the six products of parts that
// reach 2^-24 of it; what is left out stays below 2^-25.
#pragma once

#include "common.cuh"

namespace {

constexpr int kParts = 3;

// a pair of floats as three pairs of bfloat16 (the first number in the low half)
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    hi = *reinterpret_cast<uint32_t*>(&h);
    const float ra = a - __uint_as_float(hi << 16), rb = b - __uint_as_float(hi & 0xffff0000u);
    __nv_bfloat162 m = __floats2bfloat162_rn(ra, rb);
    mid = *reinterpret_cast<uint32_t*>(&m);
    __nv_bfloat162 l = __floats2bfloat162_rn(ra - __uint_as_float(mid << 16), rb - __uint_as_float(mid & 0xffff0000u));
    lo = *reinterpret_cast<uint32_t*>(&l);
}

}  // namespace
