// Portions of prompts in chunks of 64 tokens: how a block finds its (request, chunk) from the step's token offsets on the device.  The
// chunks of all requests of at least min_len tokens are numbered through in the requests' order.
#pragma once

#include "common.cuh"

namespace {

constexpr int kQ = 64;  // tokens of a chunk

struct Chunk {
    int request, start, count, slot;  // count 0: no such chunk
};

// the chunk that slot number `slot` stands for; called by a whole warp
__device__ __forceinline__ Chunk find_chunk(int slot, const int* __restrict__ qo_indptr, int n_requests, int min_len) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int b0 = 0; b0 < n_requests; b0 += 32) {
        const int b = b0 + lane;
        const int start = b < n_requests ? qo_indptr[b] : 0, len = b < n_requests ? qo_indptr[b + 1] - start : 0;
        const int chunks = len >= min_len ? (len + kQ - 1) / kQ : 0;
        int sum = chunks;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        const int c = slot - (before + sum - chunks);
        const unsigned who = __ballot_sync(0xffffffffu, c >= 0 && c < chunks);
        if (who) {
            const int src = __ffs(who) - 1;
            return {__shfl_sync(0xffffffffu, b, src), __shfl_sync(0xffffffffu, start + c * kQ, src),
                    __shfl_sync(0xffffffffu, min(kQ, len - c * kQ), src), slot};
        }
        before += __shfl_sync(0xffffffffu, sum, 31);
    }
    return {0, 0, 0, slot};
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

}  // namespace
