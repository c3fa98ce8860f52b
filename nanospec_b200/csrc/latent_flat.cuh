// Where the positions of a step's long requests lie when their cached latents are laid side by side (csrc/latent.cu gathers them, products
// unfold them, csrc/attention_prefill_tc.cu reads the result): every request of at least min_len tokens owns one row per position, from
// the block of 64 that holds the first key its first token sees to the end of the block that holds its last token, in the requests' order.
#pragma once

#include "common.cuh"

namespace {

struct FlatRows {
    int row, from, count;  // the first row, its position, and how many rows (multiples of 64)
};

// rows that request b owns, starting at position *from
__device__ __forceinline__ int flat_count(int b, const int* __restrict__ qo_indptr, const int* __restrict__ positions, int min_len, int window, int* from) {
    const int first = qo_indptr[b], len = qo_indptr[b + 1] - first;
    if (len < min_len) return 0;
    const int pos = positions[first], lo = window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0;
    *from = lo / 64 * 64;
    return (pos + len + 63) / 64 * 64 - *from;
}

// the rows of request `req`; called by a whole warp
__device__ __forceinline__ FlatRows flat_rows(int req, const int* __restrict__ qo_indptr, const int* __restrict__ positions, int min_len, int window) {
    int before = 0, from = 0;
    for (int b = threadIdx.x & 31; b < req; b += 32) before += flat_count(b, qo_indptr, positions, min_len, window, &from);
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    from = 0;
    const int count = flat_count(req, qo_indptr, positions, min_len, window, &from);
    return {before, from, count};
}

}  // namespace
