// The state space of Mamba-2 over long portions of prompts, a chunk of 64 tokens at a time instead of a token at a time.
//
// Per head, with step sizes a_t and l_t = -exp(A_log) a_t (the logarithm of the decay), L_t the sum of l over a chunk up to t and S_in the
// state before the chunk:
//     y_t   = exp(L_t) S_in^T C_t + sum_{s <= t} exp(L_t - L_s) a_s (C_t . B_s) x_s
//     S_out = exp(L_end) S_in + sum_s exp(L_end - L_s) a_s B_s x_s^T
// which is the recurrence S = exp(l) S + a B x^T, y = S^T C written out over the chunk.  Three kernels:
//     chunk_states   the sum over a chunk (a product over its tokens), every chunk and head at once, and the chunk's decay exp(L_end)
//     chunk_pass     the chunks of a request in order, element by element of the state: S_in of every chunk, and the request's state
//     chunk_outputs  y of a chunk: C B^T masked and weighted, times x, plus C S_in scaled
// Everything is float (the same operands as the token walk's: csrc/recurrent.cu), L and its differences double (or two floats), so that a
// difference of two large sums keeps its digits.  A request's chunks start at its first token of the step; requests of fewer than min_len
// tokens are left to the token walk.  Blocks find their (request, chunk) from the step's token offsets on the device.
#include <cfloat>
#include <type_traits>

#include "chunks.cuh"
#include "float_parts.cuh"
#include "mma_utils.cuh"

namespace {

constexpr int kThreads = 128;  // 8 x 16 threads on a 64 x 64 tile, 8 x 4 results each
constexpr int kLd = 68;        // floats of a staged row: 16-byte aligned, rows in different banks
constexpr int kHeads = 4;      // of a group to a block on the tensor cores

// running sums of l over the chunk (double) and the step sizes, by one warp, two tokens to a lane; tokens beyond the chunk have step 0
__device__ __forceinline__ void chunk_logs(const float* __restrict__ step, int ld, int start, int count, float a, double* L, float* dt) {
    const int lane = threadIdx.x & 31;
    const int t0 = 2 * lane, t1 = t0 + 1;
    const float d0 = t0 < count ? step[(size_t)(start + t0) * ld] : 0.f, d1 = t1 < count ? step[(size_t)(start + t1) * ld] : 0.f;
    const double l0 = -(double)(a * d0), l1 = -(double)(a * d1);
    double sum = l0 + l1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    L[t0] = sum - l1;
    L[t1] = sum;
    dt[t0] = d0;
    dt[t1] = d1;
}

// acc[8][4] += a[8] b[4]^T
__device__ __forceinline__ void outer(float (&acc)[8][4], const float4& a0, const float4& a1, const float4& b) {
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
}

// rows of a staged tile: dst[r][c] = src[(row0 + r) * ld + c] for r < rows, c < cols, zeros elsewhere, 64 x 64; `scale` (or null) per row
__device__ __forceinline__ void stage_rows(float* dst, const float* __restrict__ src, int ld, int rows, int cols, const float* scale, bool vec) {
    if (vec) {
        for (int i = threadIdx.x; i < kQ * 16; i += kThreads) {
            const int r = i >> 4, c = (i & 15) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < rows && c < cols) v = ld4(src + (size_t)r * ld + c);
            if (scale) { const float s = scale[r]; v.x *= s; v.y *= s; v.z *= s; v.w *= s; }
            *reinterpret_cast<float4*>(dst + r * kLd + c) = v;
        }
    } else {
        for (int i = threadIdx.x; i < kQ * kQ; i += kThreads) {
            const int r = i >> 6, c = i & 63;
            const float v = r < rows && c < cols ? src[(size_t)r * ld + c] : 0.f;
            dst[r * kLd + c] = scale ? v * scale[r] : v;
        }
    }
}

// grid (chunk slots, heads, tiles of 64 x 64 of the state)
__global__ void __launch_bounds__(kThreads)
chunk_states_kernel(const float* __restrict__ B, const float* __restrict__ x, const float* __restrict__ step, int ld,
                    const float* __restrict__ a_log, const int* __restrict__ qo_indptr, int n_requests, int min_len,
                    float* __restrict__ states, float* __restrict__ decays, int H, int G, int N, int Np, int V) {
    ns_pdl_launch_dependents();
    ns_pdl_wait();
    __shared__ __align__(16) float Bs[kQ * kLd], xs[kQ * kLd];
    __shared__ double L[kQ];
    __shared__ float dt[kQ], w[kQ];
    __shared__ Chunk chunk;
    const int tid = threadIdx.x, h = blockIdx.y, g = h / (H / G);
    if (tid < 32) {
        const Chunk c = find_chunk(blockIdx.x, qo_indptr, n_requests, min_len);
        if (tid == 0) chunk = c;
        if (c.count > 0) chunk_logs(step + h, ld, c.start, c.count, expf(a_log[h]), L, dt);
    }
    __syncthreads();
    const Chunk c = chunk;
    if (c.count == 0) return;
    if (tid < kQ) w[tid] = expf((float)(L[kQ - 1] - L[tid])) * dt[tid];  // (tokens beyond the chunk: step 0)
    if (tid == 0 && blockIdx.z == 0) decays[(size_t)c.slot * H + h] = expf((float)L[kQ - 1]);
    __syncthreads();
    const int v_tiles = (V + 63) / 64, n0 = (blockIdx.z / v_tiles) * 64, v0 = (blockIdx.z % v_tiles) * 64;
    stage_rows(Bs, B + (size_t)c.start * ld + (size_t)g * Np + n0, ld, c.count, N - n0, nullptr, N % 4 == 0);
    stage_rows(xs, x + (size_t)c.start * ld + (size_t)h * V + v0, ld, c.count, V - v0, w, V % 4 == 0);
    __syncthreads();
    const int ty = tid >> 4, tx = tid & 15;
    float acc[8][4] = {};
#pragma unroll 4
    for (int s = 0; s < c.count; ++s)
        outer(acc, ld4(Bs + s * kLd + ty * 8), ld4(Bs + s * kLd + ty * 8 + 4), ld4(xs + s * kLd + tx * 4));
    float* dst = states + ((size_t)c.slot * H + h) * N * V;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int n = n0 + ty * 8 + i, v = v0 + tx * 4;
        if (n >= N) break;
        if (V % 4 == 0) {
            if (v < V) *reinterpret_cast<float4*>(dst + (size_t)n * V + v) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (v + j < V) dst[(size_t)n * V + v + j] = acc[i][j];
        }
    }
}

// grid (requests, elements of the state / (256 * VEC)); states[slot] becomes the state before the chunk
template <int VEC, bool AHEAD>
__global__ void __launch_bounds__(256)
chunk_pass_kernel(float* __restrict__ states, const float* __restrict__ decays, float* __restrict__ state, long long state_floats,
                  const int* __restrict__ qo_indptr, const int* __restrict__ state_slot, int min_len, int H, int per_head) {
    ns_pdl_launch_dependents();
    ns_pdl_wait();
    __shared__ int first_slot;
    const int b = blockIdx.x, len = qo_indptr[b + 1] - qo_indptr[b];
    if (len < min_len) return;
    if (threadIdx.x < 32) {  // the chunks of the requests before this one
        int sum = 0;
        for (int r = threadIdx.x; r < b; r += 32) {
            const int n = qo_indptr[r + 1] - qo_indptr[r];
            if (n >= min_len) sum += (n + kQ - 1) / kQ;
        }
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (threadIdx.x == 0) first_slot = sum;
    }
    __syncthreads();
    const long long total = (long long)H * per_head, e = ((long long)blockIdx.y * blockDim.x + threadIdx.x) * VEC;
    if (e >= total) return;
    const int h = (int)(e / per_head), chunks = (len + kQ - 1) / kQ;  // (VEC elements lie in one head)
    float* S_mem = state + (long long)state_slot[b] * state_floats + e;
    float* at = states + (size_t)first_slot * total + e;
    const float* dec = decays + (size_t)first_slot * H + h;
    float S[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) S[k] = S_mem[k];
    // AHEAD: four chunks' loads are in flight while the four before are passed on.  What bounds this is the latency of a chain of loads (three prompts
    // of 2,471 tokens in all, 64 heads of 128 x 64: 67 us with the loads and the sums of four chunks in turn, 33 so); short prompts of few
    // heads have no chain, and the wider kernel leaves the next one's blocks less room (96 tokens, 32 heads, the whole step: 45 us in turn, 52 ahead).
    if constexpr (AHEAD) {
        float add[2][4][VEC], d[2][4];
        auto fetch = [&](int c0, int st) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c0 + u < chunks) {
                    d[st][u] = dec[(size_t)(c0 + u) * H];
                    if constexpr (VEC == 4) {
                        const float4 v = ld4(at + (size_t)(c0 + u) * total);
                        add[st][u][0] = v.x; add[st][u][1] = v.y; add[st][u][2] = v.z; add[st][u][3] = v.w;
                    } else {
                        add[st][u][0] = at[(size_t)(c0 + u) * total];
                    }
                }
        };
        auto pass = [&](int c0, int st) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (c0 + u < chunks) {
                    if constexpr (VEC == 4) *reinterpret_cast<float4*>(at + (size_t)(c0 + u) * total) = make_float4(S[0], S[1], S[2], S[3]);
                    else at[(size_t)(c0 + u) * total] = S[0];
#pragma unroll
                    for (int k = 0; k < VEC; ++k) S[k] = fmaf(d[st][u], S[k], add[st][u][k]);
                }
        };
        fetch(0, 0);
        for (int c0 = 0; c0 < chunks; c0 += 8) {
            fetch(c0 + 4, 1);
            pass(c0, 0);
            fetch(c0 + 8, 0);
            pass(c0 + 4, 1);
        }
    } else {
        for (int c0 = 0; c0 < chunks; c0 += 4) {  // four chunks' loads are in flight together
            float add[4][VEC], d[4];
            const int cnt = min(4, chunks - c0);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (u < cnt) {
                    d[u] = dec[(size_t)(c0 + u) * H];
                    if constexpr (VEC == 4) {
                        const float4 v = ld4(at + (size_t)(c0 + u) * total);
                        add[u][0] = v.x; add[u][1] = v.y; add[u][2] = v.z; add[u][3] = v.w;
                    } else {
                        add[u][0] = at[(size_t)(c0 + u) * total];
                    }
                }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (u < cnt) {
                    if constexpr (VEC == 4) *reinterpret_cast<float4*>(at + (size_t)(c0 + u) * total) = make_float4(S[0], S[1], S[2], S[3]);
                    else at[(size_t)(c0 + u) * total] = S[0];
#pragma unroll
                    for (int k = 0; k < VEC; ++k) S[k] = fmaf(d[u], S[k], add[u][k]);
                }
        }
    }
#pragma unroll
    for (int k = 0; k < VEC; ++k) S_mem[k] = S[k];
}

// grid (chunk slots, heads, tiles of 64 of a head's features)
__global__ void __launch_bounds__(kThreads, 4)
chunk_outputs_kernel(const float* __restrict__ C, const float* __restrict__ B, const float* __restrict__ x, const float* __restrict__ step,
                     int ld, const float* __restrict__ a_log, const int* __restrict__ qo_indptr, int n_requests, int min_len,
                     const float* __restrict__ states, float* __restrict__ out, int ld_out, int H, int G, int N, int Np, int V) {
    ns_pdl_launch_dependents();
    ns_pdl_wait();
    constexpr int kK = 32;  // rows of the state to a pass
    __shared__ __align__(16) float slices[3 * kK * kLd];  // C and B of the pass transposed [k][token], S_in [k][feature]; then x [token][feature]
    __shared__ __align__(16) float Mt[kQ * kLd];          // the weights of x, [s][t]
    __shared__ double L[kQ];
    __shared__ float dt[kQ];
    __shared__ Chunk chunk;
    static_assert(3 * kK >= kQ, "x takes the place of the slices");
    const int tid = threadIdx.x, h = blockIdx.y, g = h / (H / G), v0 = blockIdx.z * 64;
    if (tid < 32) {
        const Chunk c = find_chunk(blockIdx.x, qo_indptr, n_requests, min_len);
        if (tid == 0) chunk = c;
        if (c.count > 0) chunk_logs(step + h, ld, c.start, c.count, expf(a_log[h]), L, dt);
    }
    __syncthreads();
    const Chunk c = chunk;
    if (c.count == 0) return;
    const int ty = tid >> 4, tx = tid & 15;
    float *Ct = slices, *Bt = slices + kK * kLd, *Ss = slices + 2 * kK * kLd;
    const float* C0 = C + (size_t)c.start * ld + (size_t)g * Np;
    const float* B0 = B + (size_t)c.start * ld + (size_t)g * Np;
    const float* S0 = states + ((size_t)c.slot * H + h) * N * V;
    const bool vec = V % 4 == 0;
    float scores[8][4] = {}, y[8][4] = {};
    for (int k0 = 0; k0 < N; k0 += kK) {
        __syncthreads();  // the pass before has been read
        for (int i = tid; i < kQ * kK; i += kThreads) {
            const int t = i >> 5, k = i & 31;
            const bool in = t < c.count && k0 + k < N;
            Ct[k * kLd + t] = in ? C0[(size_t)t * ld + k0 + k] : 0.f;
            Bt[k * kLd + t] = in ? B0[(size_t)t * ld + k0 + k] : 0.f;
        }
        if (vec) {
            for (int i = tid; i < kK * 16; i += kThreads) {
                const int k = i >> 4, v = (i & 15) * 4;
                float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k0 + k < N && v0 + v < V) s = ld4(S0 + (size_t)(k0 + k) * V + v0 + v);
                *reinterpret_cast<float4*>(Ss + k * kLd + v) = s;
            }
        } else {
            for (int i = tid; i < kK * 64; i += kThreads) {
                const int k = i >> 6, v = i & 63;
                Ss[k * kLd + v] = k0 + k < N && v0 + v < V ? S0[(size_t)(k0 + k) * V + v0 + v] : 0.f;
            }
        }
        __syncthreads();
        const int k_end = min(kK, N - k0);
#pragma unroll 4
        for (int k = 0; k < k_end; ++k) {
            const float4 a0 = ld4(Ct + k * kLd + ty * 8), a1 = ld4(Ct + k * kLd + ty * 8 + 4);
            outer(scores, a0, a1, ld4(Bt + k * kLd + tx * 4));
            outer(y, a0, a1, ld4(Ss + k * kLd + tx * 4));
        }
    }
    // the weights of x: this thread's tokens t = 8 ty + i against s = 4 tx + j
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int s = tx * 4 + j;
        float m[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = ty * 8 + i;
            m[i] = s <= t ? scores[i][j] * (expf((float)(L[t] - L[s])) * dt[s]) : 0.f;
        }
        *reinterpret_cast<float4*>(Mt + s * kLd + ty * 8) = make_float4(m[0], m[1], m[2], m[3]);
        *reinterpret_cast<float4*>(Mt + s * kLd + ty * 8 + 4) = make_float4(m[4], m[5], m[6], m[7]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float f = expf((float)L[ty * 8 + i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) y[i][j] *= f;
    }
    __syncthreads();  // the last pass has been read; the weights are complete
    stage_rows(slices, x + (size_t)c.start * ld + (size_t)h * V + v0, ld, c.count, V - v0, nullptr, vec);
    __syncthreads();
    const int s_end = min(c.count, ((ty | 1) + 1) * 8);  // no weight of this warp's tokens lies beyond
#pragma unroll 4
    for (int s = 0; s < s_end; ++s)
        outer(y, ld4(Mt + s * kLd + ty * 8), ld4(Mt + s * kLd + ty * 8 + 4), ld4(slices + s * kLd + tx * 4));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = ty * 8 + i, v = v0 + tx * 4;
        if (t >= c.count) break;
        float* dst = out + (size_t)(c.start + t) * ld_out + (size_t)h * V + v;
        if (vec && ld_out % 4 == 0) {
            if (v < V) *reinterpret_cast<float4*>(dst) = make_float4(y[i][0], y[i][1], y[i][2], y[i][3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (v + j < V) dst[j] = y[i][j];
        }
    }
}

// ---------------------------------------------------------------------------------------
// The sums for heads of 64 features in groups of a multiple of four and states of 64 or 128 rows: a block takes four heads of a
// group, so that B is staged once for them, and threads of 8 x 8 results (16 words of shared memory to 64 FMAs; 12 to 32 above).  The same
// sums in the same order, bit for bit.  Prompts of 2,471 tokens in all, 64 heads of 64, a state of 128 rows, 8 groups: 103 us above, 77 here.
// Not on the tensor cores (66 us): a head that forgets soon has sums of a few large terms, which a chain rounds to 5.5e-8 and truncation to 7e-8.
// ---------------------------------------------------------------------------------------
constexpr int kLd4 = 68;

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int G> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(G) : "memory"); }
// a chunk's rows of COLS floats by 256 threads, zeros beyond `count`.  Every copy has an address register of its own: copies that share one wait for
// one another's data (chunk sums 81 -> 77 us)
template <int COLS>
__device__ __forceinline__ void rows_in(float* dst, int ldd, const float* __restrict__ src, int ld, int count) {
    constexpr int kPieces = COLS / 4, kCopies = kQ * kPieces / 256;
    static_assert(kQ * kPieces % 256 == 0, "a whole number of copies to a thread");
    const float* from[kCopies];
#pragma unroll
    for (int j = 0; j < kCopies; ++j) {
        const int i = threadIdx.x + j * 256, t = i / kPieces;
        from[j] = src + (size_t)(t < count ? t : 0) * ld + (i % kPieces) * 4;
    }
#pragma unroll
    for (int j = 0; j < kCopies; ++j) {
        const int i = threadIdx.x + j * 256, t = i / kPieces;
        cp_async16(dst + t * ldd + (i % kPieces) * 4, from[j], t < count);
    }
}

// acc += a b^T, 8 x 8
__device__ __forceinline__ void outer8(float (&acc)[8][8], const float4& a0, const float4& a1, const float4& b0, const float4& b1) {
    const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
}

// grid (chunk slots, H / 4), 256 threads: N / 8 x 8 threads to a head, 256 / N heads at a time
template <int N>
__global__ void __launch_bounds__(256, 2)
chunk_states4_kernel(const float* __restrict__ B, const float* __restrict__ x, const float* __restrict__ step, int ld,
                     const float* __restrict__ a_log, const int* __restrict__ qo_indptr, int n_requests, int min_len,
                     float* __restrict__ states, float* __restrict__ decays, int H, int G) {
    ns_pdl_wait();
    constexpr int kAtOnce = 256 / N, kPasses = kHeads / kAtOnce, kLdB = N + 4;
    extern __shared__ __align__(16) float states_smem[];
    float* Bs = states_smem;              // [64][N + 4]
    float* xs = Bs + kQ * kLdB;           // [kHeads][64][68]
    __shared__ double L[kHeads][kQ];
    __shared__ float dt[kHeads][kQ], w[kHeads][kQ];
    __shared__ Chunk chunk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h0 = blockIdx.y * kHeads, g = h0 / (H / G);
    if (warp == 0) {
        const Chunk c = find_chunk(blockIdx.x, qo_indptr, n_requests, min_len);
        if (lane == 0) chunk = c;
    }
    __syncthreads();
    const Chunk c = chunk;
    if (c.count == 0) return;
    const float* B0 = B + (size_t)c.start * ld + (size_t)g * N;
    rows_in<N>(Bs, kLdB, B0, ld, c.count);
    const float* x0 = x + (size_t)c.start * ld + (size_t)h0 * 64;
    for (int p = 0; p < kPasses; ++p) {  // a group of copies to a pass, so that the first heads do not wait for the others
#pragma unroll
        for (int h = p * kAtOnce; h < (p + 1) * kAtOnce; ++h) rows_in<64>(xs + h * kQ * kLd4, kLd4, x0 + h * 64, ld, c.count);
        cp_async_commit();
    }
    if (warp < kHeads) {
        const int h = h0 + warp;
        chunk_logs(step + h, ld, c.start, c.count, expf(a_log[h]), L[warp], dt[warp]);
        __syncwarp();
        for (int t = lane; t < kQ; t += 32) w[warp][t] = expf((float)(L[warp][kQ - 1] - L[warp][t])) * dt[warp][t];  // (tokens beyond the chunk: step 0)
        if (lane == 0) decays[(size_t)c.slot * H + h] = expf((float)L[warp][kQ - 1]);
    }
    const int mine = tid / N, n4 = ((tid % N) >> 3) * 4, v4 = (tid & 7) * 4;  // rows n4 .. + 3 and N / 2 + n4 .. + 3, columns v4 .. + 3 and 32 + v4 .. + 3
    for (int p = 0; p < kPasses; ++p) {
        if (kPasses == 2 && p == 0) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();
        const int hh = p * kAtOnce + mine;
        const float* xh = xs + hh * kQ * kLd4;
        float acc[8][8] = {};
#pragma unroll 2
        for (int s = 0; s < c.count; ++s) {
            const float f = w[hh][s];
            float4 b0 = ld4(xh + s * kLd4 + v4), b1 = ld4(xh + s * kLd4 + 32 + v4);
            b0.x *= f; b0.y *= f; b0.z *= f; b0.w *= f;
            b1.x *= f; b1.y *= f; b1.z *= f; b1.w *= f;
            outer8(acc, ld4(Bs + s * kLdB + n4), ld4(Bs + s * kLdB + N / 2 + n4), b0, b1);
        }
        if (p == kPasses - 1) ns_pdl_launch_dependents();
        float* dst = states + ((size_t)c.slot * H + h0 + hh) * N * 64;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float* row = dst + (size_t)((i < 4 ? n4 + i : N / 2 + n4 + i - 4)) * 64 + v4;
            *reinterpret_cast<float4*>(row) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            *reinterpret_cast<float4*>(row + 32) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
        }
    }
}

// ---------------------------------------------------------------------------------------
// The read-out for heads of 64 features with states of 64 or 128 rows on the tensor cores (m16n8k16), every float as three bfloat16 parts
// (csrc/float_parts.cuh).  What the tensor core truncates stays small: the five products with a middle or a low part have an accumulator of their
// own, the four steps of high by high of 64 k another that starts at zero, and the two and the blocks of 64 k are added rounded to nearest.
// What several heads of a group or several warps read (B, C, the weights of x) lies as parts in shared memory; x and the state lie there as floats
// and come apart on their way into the fragments of the one warp that multiplies them, a warp's columns of v dealt to its tiles in turn, so
// that a thread's are neighbours.  A block takes four heads of a group where that still makes blocks enough, or one: the same sums, bit for bit.
// Read-out of prompts of 2,471 tokens in all, 64 heads, a state of 128 rows: 191 us as FMAs, 125 here (2 of them to keep small
// operands' bits and to look for rows that are not finite); 700 tokens, 8 heads: 31.6 / 12.0.  Error of y
// against 64 bits 2.1e-7 / 1.2e-7.  Of a block's 44,000 cycles 18,000 are products (m16n8k16 at 8.2 cycles a sub-partition), 9,000 the weights of x,
// 15,000 the way to the first product; one block an SM, whose two groups of warps overlap the first two.
// ---------------------------------------------------------------------------------------
constexpr int kPadQ = 8;             // bfloat16 behind a staged row: ldmatrix reads eight rows from different banks
constexpr int kLdM = kQ + kPadQ;

// A double as the sum of two floats, and the difference of two such numbers rounded to a float: within 2^-24 (1 + 2^-20) of it, as the
// difference of the doubles rounded (what double arithmetic costs here: 12,400 of a block's 50,000 cycles).
__device__ __forceinline__ float2 two_floats(double v) {
    const float hi = (float)v;
    return make_float2(hi, isfinite(hi) ? (float)(v - (double)hi) : 0.f);
}
__device__ __forceinline__ float difference(float2 a, float2 b) {
    const float d = a.x - b.x, t = d - a.x, rest = (a.x - (d - t)) - (b.x + t);  // d + rest = a.x - b.x exactly
    return d + (rest + (a.y - b.y));
}

// three parts of a staged tile: dst[part][r][c] of src[r * ld + c], zeros from `rows` on; by 128 threads
template <int COLS>
__device__ __forceinline__ void stage_parts(__nv_bfloat16* dst, const float* __restrict__ src, int ld, int rows) {
    constexpr int kLdP = COLS + kPadQ, kEach = kQ * COLS / 4 / 128, kBatch = kEach < 16 ? kEach : 16;
    const int id = threadIdx.x & 127;
#pragma unroll 1
    for (int i0 = 0; i0 < kEach; i0 += kBatch) {  // (a batch of reads in flight)
        float4 v[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            const int i = id + (i0 + j) * 128, r = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
            v[j] = r < rows ? ld4(src + (size_t)r * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j) {
            const int i = id + (i0 + j) * 128, r = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
            uint32_t p[kParts][2];
            split_pair(v[j].x, v[j].y, p[0][0], p[1][0], p[2][0]);
            split_pair(v[j].z, v[j].w, p[0][1], p[1][1], p[2][1]);
#pragma unroll
            for (int q = 0; q < kParts; ++q) *reinterpret_cast<uint2*>(dst + (q * kQ + r) * kLdP + c) = make_uint2(p[q][0], p[q][1]);
        }
    }
}

// sums of 64 k: main takes high by high, rest the five small products
template <int MT, int NT>
struct PartSums {
    float main[MT][NT][4], rest[MT][NT][4];
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) main[i][j][e] = rest[i][j][e] = 0.f;
    }
    // row tiles I0 .. MT - 1 of A (three parts each) by all column tiles of B; neighbouring products have sums of their own
    template <int I0>
    __device__ __forceinline__ void add(const uint32_t (&a)[MT][kParts][4], const uint32_t (&b)[kParts][NT][2]) {
        constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
        for (int p = 0; p < 6; ++p)
#pragma unroll
            for (int i = I0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) ns_mma_bf16(p < 5 ? rest[i][j] : main[i][j], a[i][pa[p]], b[pb[p]][j][0], b[pb[p]][j][1]);
    }
};

// two column tiles of B from rows k = 2 q, 2 q + 1, 2 q + 8, 2 q + 9 (q = lane % 4) of a thread's two neighbouring columns
__device__ __forceinline__ void column_parts(const float2 (&v)[4], uint32_t (&b)[kParts][2][2]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        split_pair(v[2 * h].x, v[2 * h + 1].x, b[0][0][h], b[1][0][h], b[2][0][h]);
        split_pair(v[2 * h].y, v[2 * h + 1].y, b[0][1][h], b[1][1][h], b[2][1][h]);
    }
}

// A token's 16 features from the floats themselves, by one warp: what the parts cannot give (infinities, the largest numbers), and tokens that a
// later one's infinity or NaN reached through a weight of zero.  C, x, S, out: the token's, the chunk's and the head's first of these features.
template <int N>
__device__ __noinline__ void row_from_floats(const float* __restrict__ C, const float* __restrict__ B, const float* __restrict__ x,
                                             const float* __restrict__ step, int ld, float a, const float* __restrict__ S, int t, float* out) {
    const int lane = threadIdx.x & 31, f = lane & 15;
    double whole = 0.0, after[2] = {0.0, 0.0};  // of the logarithms: all up to t, those behind tokens lane and lane + 32
    for (int u = t; u >= 0; --u) {
        const double l = -(double)(a * step[(size_t)u * ld]);
        whole += l;
        if (u > lane) after[0] += l;
        if (u > lane + 32) after[1] += l;
    }
    float m[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int s = lane + 32 * j;
        if (s > t) continue;
        float z = 0.f;
        for (int n = 0; n < N; ++n) z = fmaf(C[n], B[(size_t)s * ld + n], z);
        m[j] = z * (expf((float)after[j]) * step[(size_t)s * ld]);
    }
    float y = 0.f;
    for (int n = 0; n < N; ++n) y = fmaf(C[n], S[n * 64 + f], y);
    y *= expf((float)whole);
    for (int s = 0; s <= t; ++s) y = fmaf(__shfl_sync(0xffffffffu, s < 32 ? m[0] : m[1], s & 31), x[(size_t)s * ld + f], y);
    if (lane < 16) out[f] = y;
}

// grid (chunk slots, H / HEADS): four warps to a head (64 tokens x 16 features each), HEADS / 2 heads one after the other to each of two such
// groups (one to one).  The next head's state and x come by cp.async while this one's products run: what a warp can keep in flight in
// registers is 2.4 TB/s over the GPU.
constexpr int kLdSc = kQ + 2;
template <int N, int HEADS>
struct OutputsTc {
    static constexpr int kGroups = HEADS == 1 ? 1 : 2, kThreads = kGroups * 128, kLdB = N + kPadQ;
    static constexpr int kPartsB = kParts * kQ * kLdB, kPartsM = kParts * kQ * kLdM;                       // bfloat16
    static constexpr int kShared = kPartsB > kGroups * kPartsM ? kPartsB : kGroups * kPartsM;              // B's place, then the weights'
    static constexpr int kState = N * kLd, kX = kQ * kLd;                                                  // floats of a group's staged state and x
    static constexpr int kSmem = 2 * (kPartsB + kShared) + 4 * (kQ * kLdSc + kGroups * (kState + kX));
    static_assert(kSmem + HEADS * kQ * 12 + 64 <= 227 * 1024, "shared memory");
};

template <int N, int HEADS>
__global__ void __launch_bounds__(OutputsTc<N, HEADS>::kThreads, 1)
chunk_outputs_tc_kernel(const float* __restrict__ C, const float* __restrict__ B, const float* __restrict__ x, const float* __restrict__ step,
                        int ld, const float* __restrict__ a_log, const int* __restrict__ qo_indptr, int n_requests, int min_len,
                        const float* __restrict__ states, float* __restrict__ out, int ld_out, int H, int G) {
    using O = OutputsTc<N, HEADS>;
    ns_pdl_wait();
    constexpr int kLdB = O::kLdB;
    extern __shared__ __align__(16) __nv_bfloat16 parts_smem[];
    __nv_bfloat16* Cp = parts_smem;                                   // C [part][t][n]
    __nv_bfloat16* Bp = Cp + O::kPartsB;                              // B, then the heads' weights of x [group][part][t][s]
    float* Sc = reinterpret_cast<float*>(Bp + O::kShared);            // the scores [t][s]
    __shared__ float2 Lf[HEADS][kQ];
    __shared__ float dt[HEADS][kQ];
    __shared__ Chunk chunk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, group = warp >> 2, h0 = blockIdx.y * HEADS, g = h0 / (H / G);
    if (warp == 0) {
        const Chunk c = find_chunk(blockIdx.x, qo_indptr, n_requests, min_len);
        if (lane == 0) chunk = c;
    }
    __syncthreads();
    const Chunk c = chunk;
    if (c.count == 0) return;
    float* Ss = Sc + kQ * kLdSc + group * (O::kState + O::kX);        // this group's state [n][v] and x [t][v]
    float* Xs = Ss + O::kState;
    const int id = tid & 127;
    auto load_state = [&](int hh) {
        const float* src = states + ((size_t)c.slot * H + h0 + hh) * N * 64;
        for (int i = id; i < N * 16; i += 128) cp_async16(Ss + (i >> 4) * kLd + (i & 15) * 4, src + i * 4, true);
        cp_async_commit();
    };
    auto load_x = [&](int hh) {
        const float* src = x + (size_t)c.start * ld + (size_t)(h0 + hh) * 64;
        for (int i = id; i < kQ * 16; i += 128) {
            const int t = i >> 4;
            cp_async16(Xs + t * kLd + (i & 15) * 4, src + (size_t)(t < c.count ? t : 0) * ld + (i & 15) * 4, t < c.count);
        }
        cp_async_commit();
    };
    auto group_sync = [&] { asm volatile("bar.sync %0, 128;" ::"r"(1 + group) : "memory"); };
    load_state(group);
    load_x(group);
    // one group C, the other B and the logarithms
    if (group == 0) stage_parts<N>(Cp, C + (size_t)c.start * ld + (size_t)g * N, ld, c.count);
    if (group == O::kGroups - 1) {
        if ((warp & 3) < HEADS) {
            const int hh = warp & 3;
            double* L = reinterpret_cast<double*>(Sc) + hh * kQ;  // (the scores come later)
            chunk_logs(step + h0 + hh, ld, c.start, c.count, expf(a_log[h0 + hh]), L, dt[hh]);
            __syncwarp();
            for (int t = lane; t < kQ; t += 32) Lf[hh][t] = two_floats(L[t]);
        }
        stage_parts<N>(Bp, B + (size_t)c.start * ld + (size_t)g * N, ld, c.count);
    }
    __syncthreads();
    const int q = lane & 3, quad = lane >> 2, mi = lane >> 3, t0 = (warp & 3) * 16;
    const __nv_bfloat16* c_at = Cp + (lane & 15) * kLdB + (lane >> 4) * 8;  // of ldmatrix: row t, column n of C
    // the scores: 16 tokens t by 32 tokens s to a warp
    for (int sh = group; sh < 2; sh += O::kGroups) {
        float total[4][4] = {};
        if (sh * 32 <= t0) {  // (the others are masked)
#pragma unroll 1
            for (int kb = 0; kb < N; kb += 64) {
                PartSums<1, 4> z;
                z.clear();
#pragma unroll
                for (int k0 = 0; k0 < 64; k0 += 16) {
                    uint32_t a[1][kParts][4], b[kParts][4][2];
#pragma unroll
                    for (int p = 0; p < kParts; ++p) {
                        ns_ldmatrix_x4(a[0][p], c_at + (p * kQ + t0) * kLdB + kb + k0);
#pragma unroll
                        for (int j = 0; j < 4; j += 2) {
                            uint32_t r[4];
                            ns_ldmatrix_x4(r, Bp + (p * kQ + sh * 32 + j * 8 + (mi >> 1) * 8 + (lane & 7)) * kLdB + kb + k0 + (mi & 1) * 8);
                            b[p][j][0] = r[0]; b[p][j][1] = r[1]; b[p][j + 1][0] = r[2]; b[p][j + 1][1] = r[3];
                        }
                    }
                    z.add<0>(a, b);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) total[j][e] += z.main[0][j][e] + z.rest[0][j][e];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r)
                *reinterpret_cast<float2*>(Sc + (t0 + quad + 8 * r) * kLdSc + sh * 32 + j * 8 + 2 * q) = make_float2(total[j][2 * r] * kPartsBack, total[j][2 * r + 1] * kPartsBack);
    }
    __syncthreads();  // the scores are there, B has been read
    const int v0 = (warp & 3) * 16, steps = (c.count + 15) >> 4;
    __nv_bfloat16* Mp = Bp + group * O::kPartsM;
    const __nv_bfloat16* m_at = Mp + (lane & 15) * kLdM + (lane >> 4) * 8;
    const float *s_at = Ss + 2 * q * kLd + v0 + quad * 2, *x_at = Xs + 2 * q * kLd + v0 + quad * 2;
    auto columns = [&](const float* at, int k0, uint32_t (&b)[kParts][2][2]) {  // rows k0 + 2 q, + 1, + 8, + 9 of a thread's two columns
        float2 v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = *reinterpret_cast<const float2*>(at + (k0 + (e & 1) + (e >> 1) * 8) * kLd);
        column_parts(v, b);
    };
    unsigned odd = 0;  // bit by head: something that this thread wrote is not finite
#pragma unroll 1
    for (int hh = group; hh < HEADS; hh += O::kGroups) {
        const int h = h0 + hh;
        const bool more = hh + O::kGroups < HEADS;
        float y[4][2][4] = {};
        PartSums<4, 2> sums;
        auto take = [&] {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) y[i][j][e] += sums.main[i][j][e] + sums.rest[i][j][e];
        };
        // the weights of x: a warp 16 tokens t, a lane two tokens s
        auto weights = [&] {
            constexpr int kBatch = 8;
            const float2 l0 = Lf[hh][2 * lane], l1 = Lf[hh][2 * lane + 1];
            const float d0 = dt[hh][2 * lane], d1 = dt[hh][2 * lane + 1];
#pragma unroll 1
            for (int r0 = 0; r0 < 16; r0 += kBatch) {  // (reads first, writes last: in turn each row would wait for the one before)
                float2 z[kBatch], lt[kBatch];
                uint32_t p[kBatch][kParts];
#pragma unroll
                for (int r = 0; r < kBatch; ++r) {
                    z[r] = *reinterpret_cast<const float2*>(Sc + (t0 + r0 + r) * kLdSc + 2 * lane);
                    lt[r] = Lf[hh][t0 + r0 + r];
                }
#pragma unroll
                for (int r = 0; r < kBatch; ++r) {
                    const bool in0 = 2 * lane <= t0 + r0 + r, in1 = 2 * lane + 1 <= t0 + r0 + r;
                    const float e0 = expf(in0 ? difference(lt[r], l0) : 0.f), e1 = expf(in1 ? difference(lt[r], l1) : 0.f);  // (of all lanes: no branch)
                    split_pair(in0 ? z[r].x * (e0 * d0) : 0.f, in1 ? z[r].y * (e1 * d1) : 0.f, p[r][0], p[r][1], p[r][2]);
                }
#pragma unroll
                for (int r = 0; r < kBatch; ++r)
#pragma unroll
                    for (int k = 0; k < kParts; ++k) *reinterpret_cast<uint32_t*>(Mp + (k * kQ + t0 + r0 + r) * kLdM + 2 * lane) = p[r][k];
            }
        };
        // The first group makes its weights before C S_in, the second after it: one is on the CUDA cores while the other is on the tensor cores.
        if (group == 0) weights();
        cp_async_wait<0>();
        group_sync();  // the head's state and x are there
        // C S_in
#pragma unroll 1
        for (int kb = 0; kb < N; kb += 64) {
            sums.clear();
#pragma unroll
            for (int k = 0; k < 64; k += 16) {
                uint32_t a[4][kParts][4], b[kParts][2][2];
                columns(s_at, kb + k, b);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int p = 0; p < kParts; ++p) ns_ldmatrix_x4(a[i][p], c_at + (p * kQ + i * 16) * kLdB + kb + k);
                sums.template add<0>(a, b);
            }
            take();
        }
        if (group == 1) weights();
        group_sync();  // the state has been read, the weights are there
        if (more) load_state(hh + O::kGroups);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const float f = expf(Lf[hh][i * 16 + quad + 8 * r].x);
#pragma unroll
                for (int j = 0; j < 2; ++j) { y[i][j][2 * r] *= f; y[i][j][2 * r + 1] *= f; }
            }
        // the weights times x; a row tile ends at its own tokens
        sums.clear();
        auto row_tiles = [&](auto first_tile) {  // tokens 16 KS .. + 15 of x, for row tiles KS .. 3
            constexpr int KS = decltype(first_tile)::value;
            if (KS >= steps) return;
            uint32_t a[4][kParts][4], b[kParts][2][2];
            columns(x_at, KS * 16, b);
#pragma unroll
            for (int i = KS; i < 4; ++i)
#pragma unroll
                for (int p = 0; p < kParts; ++p) ns_ldmatrix_x4(a[i][p], m_at + (p * kQ + i * 16) * kLdM + KS * 16);
            sums.template add<KS>(a, b);
        };
        row_tiles(std::integral_constant<int, 0>{});
        row_tiles(std::integral_constant<int, 1>{});
        row_tiles(std::integral_constant<int, 2>{});
        row_tiles(std::integral_constant<int, 3>{});
        take();
        if (more) {
            group_sync();  // x and the weights have been read
            load_x(hh + O::kGroups);
        } else {
            ns_pdl_launch_dependents();
        }
        float zero = 0.f;  // as long as everything is finite
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = i * 16 + quad + 8 * r;
                const float4 v = make_float4(y[i][0][2 * r] * kPartsBack, y[i][1][2 * r] * kPartsBack, y[i][0][2 * r + 1] * kPartsBack,
                                             y[i][1][2 * r + 1] * kPartsBack);
                if (t < c.count) *reinterpret_cast<float4*>(out + (size_t)(c.start + t) * ld_out + (size_t)h * 64 + v0 + q * 4) = v;
                zero = fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, zero))));
            }
        odd |= (unsigned)(zero != 0.f) << hh;
    }
    odd = __reduce_or_sync(0xffffffffu, odd);
#pragma unroll 1
    for (; odd; odd &= odd - 1) {  // rows that are not finite, from the floats
        const int h = h0 + __ffs(odd) - 1;
#pragma unroll 1
        for (int k = 0; k < 8; ++k) {
            const int first = (k >> 1) * 16 + 8 * (k & 1);
            bool mine = false;
            if (first + quad < c.count) {
                const float4 v = *reinterpret_cast<const float4*>(out + (size_t)(c.start + first + quad) * ld_out + (size_t)h * 64 + v0 + q * 4);
                mine = !(fabsf(v.x + v.y + (v.z + v.w)) <= FLT_MAX);  // (numbers are below 2^80 here: their sum is one)
            }
            for (unsigned who = __ballot_sync(0xffffffffu, mine); who;) {
                const int row = (__ffs(who) - 1) >> 2, t = first + row;
                who &= ~(15u << (4 * row));
                row_from_floats<N>(C + (size_t)(c.start + t) * ld + (size_t)g * N, B + (size_t)c.start * ld + (size_t)g * N,
                                   x + (size_t)c.start * ld + (size_t)h * 64 + v0, step + (size_t)c.start * ld + h, ld, expf(a_log[h]),
                                   states + ((size_t)c.slot * H + h) * N * 64 + v0, t, out + (size_t)(c.start + t) * ld_out + (size_t)h * 64 + v0);
            }
        }
    }
}

template <int N>
int launch_states4(const float* B, const float* x, const float* step, int ld, const float* a_log, const int* qo_indptr, int n_requests, int min_len,
                   int chunks, float* states, float* decays, int H, int G, cudaStream_t stream) {
    constexpr int smem = 4 * (kQ * (N + 4) + kHeads * kQ * kLd4);
    NS_CUDA(cudaFuncSetAttribute(chunk_states4_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    NS_LAUNCH(chunk_states4_kernel<N>, dim3(chunks, H / kHeads), 256, smem, stream, B, x, step, ld, a_log, qo_indptr, n_requests, min_len, states, decays, H, G);
    NS_CHECK_LAUNCH("ns_ssm_chunked");
    return NS_OK;
}
template <int N, int HEADS>
int launch_outputs_tc(const float* C, const float* B, const float* x, const float* step, int ld, const float* a_log, const int* qo_indptr, int n_requests,
                      int min_len, int chunks, const float* states, float* out, int ld_out, int H, int G, cudaStream_t stream) {
    using O = OutputsTc<N, HEADS>;
    NS_CUDA(cudaFuncSetAttribute(chunk_outputs_tc_kernel<N, HEADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, O::kSmem));
    NS_LAUNCH((chunk_outputs_tc_kernel<N, HEADS>), dim3(chunks, H / HEADS), O::kThreads, O::kSmem, stream, C, B, x, step, ld, a_log, qo_indptr, n_requests,
              min_len, states, out, ld_out, H, G);
    NS_CHECK_LAUNCH("ns_ssm_chunked");
    return NS_OK;
}

}  // namespace

// C, B, x, step: the columns of the preparation's rows (row stride ld floats; groups of C and B Np apart, heads of x V, one step size
// per head); a_log [H]; state [slots, state_floats] with S [H, N, V] at the start of a row; states: scratch for `chunks` chunks of
// H * N * V floats, decays: H floats each, where `chunks` is at least the number of chunks of all requests of min_len tokens or more.
// Requests of fewer tokens are not touched.  Four heads go to a block, where they can, once that makes more than
// `four_from` blocks (half of that on the tensor cores).
NS_API int ns_ssm_chunked(const float* C, const float* B, const float* x, const float* step, int ld, const float* a_log, float* state,
                          long long state_floats, const int* qo_indptr, const int* state_slot, float* out, int ld_out, int n_requests,
                          int min_len, int chunks, float* states, float* decays, int H, int G, int N, int Np, int V, int four_from, cudaStream_t stream) {
    if (n_requests <= 0 || chunks <= 0) return NS_OK;
    if (G < 1 || H % G || N < 1 || V < 1 || Np < N) NS_FAIL(NS_ERR_ARGUMENT, "ns_ssm_chunked: %d heads in %d groups, state %d (%d), features %d", H, G, N, Np, V);
    if (ld % 4 || Np % 4 || (((uintptr_t)C | (uintptr_t)B | (uintptr_t)x | (uintptr_t)states) % 16) || (V % 4 == 0 && (uintptr_t)out % 16))
        NS_FAIL(NS_ERR_ARGUMENT, "ns_ssm_chunked: rows must start on 16 bytes");
    const int n_tiles = (N + 63) / 64, v_tiles = (V + 63) / 64;
    if (H > 65535 || n_tiles * v_tiles > 65535) NS_FAIL(NS_ERR_UNSUPPORTED, "ns_ssm_chunked: %d heads, state of %d x %d exceed the grid", H, N, V);
    const bool many = (long long)chunks * H > (long long)four_from * kHeads;
    const bool tensor = V == 64 && (N == 64 || N == 128) && Np == N && ld_out % 4 == 0, group4 = tensor && (H / G) % kHeads == 0, four = many && group4;
    if (four) {
        auto* launch = N == 128 ? launch_states4<128> : launch_states4<64>;
        const int rc = launch(B, x, step, ld, a_log, qo_indptr, n_requests, min_len, chunks, states, decays, H, G, stream);
        if (rc) return rc;
    } else {
        NS_LAUNCH(chunk_states_kernel, dim3(chunks, H, n_tiles * v_tiles), kThreads, 0, stream, B, x, step, ld, a_log, qo_indptr, n_requests, min_len,
                  states, decays, H, G, N, Np, V);
    }
    NS_CHECK_LAUNCH("ns_ssm_chunked");
    const long long total = (long long)H * N * V;
    const bool vec = (N * V) % 4 == 0 && state_floats % 4 == 0 && (uintptr_t)state % 16 == 0;
    const long long blocks = (total + 256 * (vec ? 4 : 1) - 1) / (256 * (vec ? 4 : 1));
    if (blocks > 65535) NS_FAIL(NS_ERR_UNSUPPORTED, "ns_ssm_chunked: a state of %lld floats exceeds the grid", total);
#define NS_SSM_PASS(VC, AH)                                                                                                                \
    NS_LAUNCH((chunk_pass_kernel<VC, AH>), dim3(n_requests, (unsigned)blocks), 256, 0, stream, states, decays, state, state_floats, qo_indptr, \
              state_slot, min_len, H, N * V)
    if (vec) { if (many) NS_SSM_PASS(4, true); else NS_SSM_PASS(4, false); }
    else { if (many) NS_SSM_PASS(1, true); else NS_SSM_PASS(1, false); }
#undef NS_SSM_PASS
    NS_CHECK_LAUNCH("ns_ssm_chunked");
    if (tensor) {
        // a round of blocks of four heads takes 24 us with a state of 128 rows, one of a head each 11.7: four from two rounds of single heads on (500
        // tokens, 64 heads: 24 against 47 us; 150 tokens, 32 heads: 22 against 12)
        const bool fours = group4 && (long long)chunks * H > 2LL * four_from;
        auto* launch = N == 128 ? (fours ? launch_outputs_tc<128, kHeads> : launch_outputs_tc<128, 1>)
                                : (fours ? launch_outputs_tc<64, kHeads> : launch_outputs_tc<64, 1>);
        return launch(C, B, x, step, ld, a_log, qo_indptr, n_requests, min_len, chunks, states, out, ld_out, H, G, stream);
    }
    NS_LAUNCH(chunk_outputs_kernel, dim3(chunks, H, v_tiles), kThreads, 0, stream, C, B, x, step, ld, a_log, qo_indptr, n_requests, min_len,
              states, out, ld_out, H, G, N, Np, V);
    NS_CHECK_LAUNCH("ns_ssm_chunked");
    return NS_OK;
}
