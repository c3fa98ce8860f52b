// Retention and the gated delta rule (csrc/recurrent.cu) over long portions of prompts, a chunk of 64 tokens at a time.
//
// Per head, with l_t the logarithm of the decay, L_t its sum over the chunk up to t, e_t = exp(L_t), S_in the state before the chunk, and
// the rows u_t that the tokens write (S_t = exp(l_t) S_(t-1) + k_t u_t^T):
//     u_t = v_t                                                                         retention
//     u_t = beta_t (v_t - e_t S_in^T k_t - sum_{s < t} exp(L_t - L_s) (k_t . k_s) u_s)  delta rule
//     o_t = e_t S_in^T q_t + sum_{s <= t} exp(L_t - L_s) (q_t . k_s) u_s
//     S_out = e_end S_in + sum_s exp(L_end - L_s) k_s u_s^T
// The delta rule's u solve (I + A) U = beta V - (beta e K) S_in with A strictly lower triangular, so with T = (I + A)^-1
//     U = T (beta V) - W S_in,   W = T (beta e K)
// and only the products with S_in wait for the chunk before.  Three kernels:
//     chunk_solve    every chunk and head at once: A, T (blocks of 16 by substitution, joined by products), W and T (beta V)
//     chunk_walk     the chunks of a request in order, 16 columns of S to a block: U, S_out, and S_in left for the next kernel
//     chunk_read     every chunk and head at once: the read-out
// A weight that the masks above leave out is skipped, not multiplied as a zero: a NaN or an infinity of one token stays out of the tokens
// before it, as in the walk by token.
// Everything is float, L and its differences double; products are fp32 FMAs on the CUDA cores.  The products' bound is what shared
// memory can return: 12 words to 32 FMAs a thread (8 x 4 tiles).  The kernels let their successor in when their products are done (blocks
// placed earlier would land unevenly).
#include "chunks.cuh"

namespace {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc[i][j] += a_i . b_j over four k: rows a + 4 i lda and b + 8 j ldb
template <int TM, int TN>
__device__ __forceinline__ void fma_rows(float (&acc)[TM][TN], const float* a, int lda, const float* b, int ldb) {
    float4 bv[TN];
#pragma unroll
    for (int j = 0; j < TN; ++j) bv[j] = ld4(b + 8 * j * ldb);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const float4 av = ld4(a + 4 * i * lda);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            acc[i][j] = fmaf(av.x, bv[j].x, acc[i][j]);
            acc[i][j] = fmaf(av.y, bv[j].y, acc[i][j]);
            acc[i][j] = fmaf(av.z, bv[j].z, acc[i][j]);
            acc[i][j] = fmaf(av.w, bv[j].w, acc[i][j]);
        }
    }
}

// acc += a . b over n k (a multiple of 32): runs of 32 summed by themselves, so that no chain of roundings is longer
template <int TM, int TN>
__device__ __forceinline__ void dot_rows(float (&acc)[TM][TN], const float* a, int lda, const float* b, int ldb, int n) {
    for (int e0 = 0; e0 < n; e0 += 32) {
        float run[TM][TN] = {};
#pragma unroll 4
        for (int e = e0; e < e0 + 32; e += 4) fma_rows<TM, TN>(run, a + e, lda, b + e, ldb);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] += run[i][j];
    }
}

// L of the chunk's tokens by one warp, two to a lane; tokens beyond the chunk do not decay.  `gate`: decays per token (row stride ld), or
// null: `fixed`.  A decay of 0 counts as exp(-200), whose float is 0, so that differences stay numbers; one that is no number, or negative, has no
// logarithm and makes what it enters a NaN.
__device__ __forceinline__ void gate_logs(const float* __restrict__ gate, int ld, float fixed, int start, int count, double* L) {
    const int lane = threadIdx.x & 31, t0 = 2 * lane, t1 = t0 + 1;
    auto log_of = [&](int t) {
        const float g = t >= count ? 1.f : gate ? gate[(size_t)(start + t) * ld] : fixed;
        return g == 0.f ? -200.0 : log((double)g);
    };
    const double l0 = log_of(t0), l1 = log_of(t1);
    double sum = l0 + l1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
    }
    const double before = __shfl_up_sync(0xffffffffu, sum, 1);
    L[t0] = lane ? before + l0 : l0;  // (not sum - l1, which a later token's infinity would make a NaN)
    L[t1] = sum;
}

// x[t][e] = src[(start + t) * ld + e] for t < count, zeros beyond; COLS floats to a row, `ldx` apart.  Every copy has an address register of its own:
// copies that share one wait for one another's data (reads of a prompt of 2,048 tokens 79 -> 75 us)
template <int THREADS, int COLS>
__device__ __forceinline__ void stage(float* x, int ldx, const float* __restrict__ src, int ld, int count) {
    constexpr int kPieces = COLS / 4, kCopies = (kQ * kPieces + THREADS - 1) / THREADS;
    const float* from[kCopies];
#pragma unroll
    for (int j = 0; j < kCopies; ++j) {
        const int i = threadIdx.x + j * THREADS, t = i / kPieces;
        from[j] = src + (size_t)(t < count ? t : 0) * ld + (i - t * kPieces) * 4;
    }
#pragma unroll
    for (int j = 0; j < kCopies; ++j) {
        const int i = threadIdx.x + j * THREADS, t = i / kPieces;
        if (kQ * kPieces % THREADS == 0 || t < kQ) cp_async16(x + t * ldx + (i - t * kPieces) * 4, from[j], t < count);
    }
}

// ---------------------------------------------------------------------------------------
// grid (chunk slots, heads), 256 threads.  W [slot, head, 64, D], U [slot, head, 64, V]; fade [slot, head, 64]: exp(L_end - L_t);
// whole [slot, head]: exp(L_end).  k null (retention): fade and whole alone.
// ---------------------------------------------------------------------------------------
constexpr int kLdT = kQ + 4;

template <int D>
__global__ void __launch_bounds__(256)
chunk_solve_kernel(const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ gate, const float* __restrict__ beta,
                   const float* __restrict__ decay, int ld, const int* __restrict__ qo_indptr, int n_requests, int min_len,
                   float* __restrict__ W, float* __restrict__ U, float* __restrict__ fade, float* __restrict__ whole, int H, int G, int V) {
    ns_pdl_wait();
    constexpr int kLdK = D + 4, kCols = 128, kLdV = kCols + 4;
    extern __shared__ __align__(16) float solve_smem[];
    float* Ks = solve_smem;             // [64][D + 4]
    float* Vs = Ks + kQ * kLdK;         // [64][128 + 4]
    float* As = Vs + kQ * kLdV;         // [64][68]
    float* Ts = As + kQ * kLdT;         // [64][68]
    float* tmp = Ts + kQ * kLdT;        // [3][16][17]
    __shared__ double L[kQ];
    __shared__ float bt[kQ];
    __shared__ Chunk chunk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y;
    if (warp == 0) {
        const Chunk c = find_chunk(blockIdx.x, qo_indptr, n_requests, min_len);
        if (lane == 0) chunk = c;
        if (c.count > 0) gate_logs(gate ? gate + h : nullptr, ld, decay ? decay[h] : 1.f, c.start, c.count, L);
    }
    __syncthreads();
    const Chunk c = chunk;
    if (c.count == 0) return;
    const size_t item = (size_t)c.slot * H + h;
    if (tid < kQ) fade[item * kQ + tid] = expf((float)(L[kQ - 1] - L[tid]));
    if (tid == 0) whole[item] = expf((float)L[kQ - 1]);
    if (!k) return;
    const float* k0 = k + (size_t)c.start * ld + (size_t)(h / (H / G)) * D;
    const float* v0 = v + (size_t)c.start * ld + (size_t)h * V;
    stage<256, D>(Ks, kLdK, k0, ld, c.count);
    cp_async_commit();
    if (tid < kQ) bt[tid] = tid < c.count ? beta[(size_t)(c.start + tid) * ld + h] : 0.f;
    cp_async_wait<0>();
    __syncthreads();
    // A: three warps, a lower 32 x 32 block each; the others clear T
    if (warp < 3) {
        const int tr = warp ? 32 : 0, sc = warp == 2 ? 32 : 0, ly = lane >> 3, lx = lane & 7;
        float acc[8][4] = {};
        dot_rows<8, 4>(acc, Ks + (tr + ly) * kLdK, kLdK, Ks + (sc + lx) * kLdK, kLdK, D);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = tr + ly + 4 * i, s = sc + lx + 8 * j;
                As[t * kLdT + s] = s < t ? bt[t] * expf((float)(L[t] - L[s])) * acc[i][j] : 0.f;
            }
    } else {
        for (int i = tid - 96; i < kQ * kLdT / 4; i += 160) *reinterpret_cast<float4*>(Ts + 4 * i) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    // the rows of the right-hand sides; T's diagonal blocks, a column to a thread
    for (int i = tid; i < kQ * (D / 4); i += 256) {
        const int t = i / (D / 4), e = (i % (D / 4)) * 4;
        const float f = bt[t] * expf((float)L[t]);
        float4 x = ld4(Ks + t * kLdK + e);
        x.x *= f; x.y *= f; x.z *= f; x.w *= f;
        *reinterpret_cast<float4*>(Ks + t * kLdK + e) = x;
    }
    if (tid < kQ) {
        const int b = (tid >> 4) * 16, j = tid & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float sum = 0.f;
#pragma unroll
            for (int s = 0; s < 16; ++s)
                if (s < i) sum = fmaf(As[(b + i) * kLdT + b + s], x[s], sum);
            x[i] = i == j ? 1.f : i < j ? 0.f : -sum;
            Ts[(b + i) * kLdT + b + j] = x[i];
        }
    }
    __syncthreads();
    // block (bi, bi - off) of T: -T(bi, bi) sum_k A(bi, k) T(k, bi - off)
    const int r = tid >> 4, cc = tid & 15;
    for (int off = 1; off < 4; ++off) {
        for (int n = 0; n < 4 - off; ++n) {
            const int bi = n + off, bj = n;
            float sum = 0.f;
            for (int kk = bj * 16; kk < bi * 16; ++kk) sum = fmaf(As[(bi * 16 + r) * kLdT + kk], Ts[kk * kLdT + bj * 16 + cc], sum);
            tmp[(n * 16 + r) * 17 + cc] = sum;
        }
        __syncthreads();
        for (int n = 0; n < 4 - off; ++n) {
            const int bi = n + off, bj = n;
            float sum = 0.f;
#pragma unroll
            for (int kk = 0; kk < 16; ++kk)
                if (kk <= r) sum = fmaf(Ts[(bi * 16 + r) * kLdT + bi * 16 + kk], tmp[(n * 16 + kk) * 17 + cc], sum);
            Ts[(bi * 16 + r) * kLdT + bj * 16 + cc] = -sum;
        }
        __syncthreads();
    }
    // T times a right-hand side of up to 128 columns: warp w the rows 8 w .. 8 w + 7, a lane four columns
    auto product = [&](const float* x, int ldx, int cols, float* dst, int ld_dst) {
        if (lane * 4 < cols) {
            float acc[8][4] = {};
            auto add = [&](int s, int first) {  // columns s .. s + 3 of T; in the diagonal block row i ends at its own column, first + i
                float4 b[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) b[u] = ld4(x + (s + u) * ldx + lane * 4);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (first + i < 0) continue;
                    const float4 a = ld4(Ts + (8 * warp + i) * kLdT + s);
                    const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (u > first + i) break;
                        acc[i][0] = fmaf(av[u], b[u].x, acc[i][0]);
                        acc[i][1] = fmaf(av[u], b[u].y, acc[i][1]);
                        acc[i][2] = fmaf(av[u], b[u].z, acc[i][2]);
                        acc[i][3] = fmaf(av[u], b[u].w, acc[i][3]);
                    }
                }
            };
            for (int s = 0; s < 8 * warp; s += 4) add(s, 3);
            add(8 * warp, 0);
            add(8 * warp + 4, -4);
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float4*>(dst + (size_t)(8 * warp + i) * ld_dst + lane * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
    };
    product(Ks, kLdK, D, W + item * kQ * D, D);
    ns_pdl_launch_dependents();
    for (int e0 = 0; e0 < V; e0 += kCols) {
        const int cols = min(kCols, V - e0);
        __syncthreads();
        for (int i = tid; i < kQ * (cols / 4); i += 256) {
            const int t = i / (cols / 4), e = (i % (cols / 4)) * 4;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t < c.count) {
                x = ld4(v0 + (size_t)t * ld + e0 + e);
                x.x *= bt[t]; x.y *= bt[t]; x.z *= bt[t]; x.w *= bt[t];
            }
            *reinterpret_cast<float4*>(Vs + t * kLdV + e) = x;
        }
        __syncthreads();
        product(Vs, kLdV, cols, U + item * kQ * V + e0, V);
    }
}

// ---------------------------------------------------------------------------------------
// grid (requests, heads, V / 16), 2 D threads.  S lies transposed in shared memory, [column][row].  Per chunk
//     U = U0 - W S     a lane an eighth of the rows of S (float4 pieces, interleaved), tiles of 8 tokens x 4 columns, eight lanes' sums joined
//     S = e S + K^T U  a lane a quarter of the tokens, tiles of 8 rows x 4 columns, four lanes' sums joined
// with the next chunk's W, K and U0 on their way.  states [slot, head, V, D]: S before the chunk.
// ---------------------------------------------------------------------------------------
constexpr int kVC = 16;

template <int D, bool DELTA>
__global__ void __launch_bounds__(2 * D)
chunk_walk_kernel(const float* __restrict__ k, const float* __restrict__ v, int ld, const float* __restrict__ W, float* __restrict__ U,
                  const float* __restrict__ fade, const float* __restrict__ whole, float* __restrict__ states, float* __restrict__ state,
                  long long state_floats, const int* __restrict__ qo_indptr, const int* __restrict__ state_slot, int min_len, int H, int G, int V) {
    ns_pdl_wait();
    constexpr int kThreads = 2 * D, kWarps = kThreads / 32, kLdS = D + 4, kLdU = kVC + 4;
    constexpr int kStage = kQ * D * (DELTA ? 2 : 1) + kQ * kVC;
    extern __shared__ __align__(16) float walk_smem[];
    float* St = walk_smem;                  // [16][D + 4]
    float* Us = St + kVC * kLdS;            // [64][20]: the rows u times their fade
    float* stages = Us + kQ * kLdU;         // two of K [64][D], U0 [64][16], W [64][D]
    __shared__ float fs[2][kQ], es[2];
    __shared__ int first_slot;
    const int b = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * kVC;
    const int start = qo_indptr[b], len = qo_indptr[b + 1] - start;
    if (len < min_len) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (warp == 0) {  // the chunks of the requests before this one
        int sum = 0;
        for (int r = lane; r < b; r += 32) {
            const int n = qo_indptr[r + 1] - qo_indptr[r];
            if (n >= min_len) sum += (n + kQ - 1) / kQ;
        }
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) first_slot = sum;
    }
    float* S_mem = state + (long long)state_slot[b] * state_floats + (long long)h * D * V + v0;
    for (int i = tid; i < D * kVC; i += kThreads) St[(i % kVC) * kLdS + i / kVC] = S_mem[(size_t)(i / kVC) * V + i % kVC];
    __syncthreads();
    const int chunks = (len + kQ - 1) / kQ;
    const float* kh = k + (size_t)(h / (H / G)) * D;

    auto issue = [&](int c) {
        if (c < chunks) {
            float* st = stages + (c & 1) * kStage;
            const size_t item = (size_t)(first_slot + c) * H + h;
            const int n0 = start + c * kQ, count = min(kQ, len - c * kQ);
            stage<kThreads, D>(st, D, kh + (size_t)n0 * ld, ld, count);
            if (DELTA) {
                stage<kThreads, kVC>(st + kQ * D, kVC, U + item * kQ * V + v0, V, kQ);
                stage<kThreads, D>(st + kQ * D + kQ * kVC, D, W + item * kQ * D, D, kQ);
            } else {
                stage<kThreads, kVC>(st + kQ * D, kVC, v + (size_t)n0 * ld + (size_t)h * V + v0, ld, count);
            }
            if (tid < kQ) fs[c & 1][tid] = fade[item * kQ + tid];
            if (tid == 0) es[c & 1] = whole[item];
        }
        cp_async_commit();
    };
    issue(0);
    for (int c = 0; c < chunks; ++c) {
        issue(c + 1);
        cp_async_wait<1>();
        __syncthreads();  // chunk c is there, and S is complete
        const float* Kc = stages + (c & 1) * kStage;
        const float* U0 = Kc + kQ * D;
        const size_t item = (size_t)(first_slot + c) * H + h;
        float* Sg = states + (item * V + v0) * D;
        for (int i = tid; i < kVC * (D / 4); i += kThreads) {
            const int col = i / (D / 4), e = (i % (D / 4)) * 4;
            *reinterpret_cast<float4*>(Sg + (size_t)col * D + e) = ld4(St + col * kLdS + e);
        }
        if (DELTA) {
            const float* Wc = U0 + kQ * kVC;
            const int part = lane & 7, cg = (lane >> 3) * 4;
            for (int tq = warp; tq < 8; tq += kWarps) {
                float acc[8][4] = {};
#pragma unroll
                for (int e = 4 * part; e < D; e += 32) {
                    float4 s[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[j] = ld4(St + (cg + j) * kLdS + e);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float4 w = ld4(Wc + (tq * 8 + i) * D + e);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            acc[i][j] = fmaf(w.x, s[j].x, acc[i][j]);
                            acc[i][j] = fmaf(w.y, s[j].y, acc[i][j]);
                            acc[i][j] = fmaf(w.z, s[j].z, acc[i][j]);
                            acc[i][j] = fmaf(w.w, s[j].w, acc[i][j]);
                        }
                    }
                }
                // the eight lanes' sums: after the three exchanges a lane holds one token's
                float a4[4][4], a2[2][4], a1[4];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool up = part & 4;
                        const float keep = up ? acc[i + 4][j] : acc[i][j], give = up ? acc[i][j] : acc[i + 4][j];
                        a4[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, 4);
                    }
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const bool up = part & 2;
                        const float keep = up ? a4[i + 2][j] : a4[i][j], give = up ? a4[i][j] : a4[i + 2][j];
                        a2[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
                    }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const bool up = part & 1;
                    const float keep = up ? a2[1][j] : a2[0][j], give = up ? a2[0][j] : a2[1][j];
                    a1[j] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
                }
                const int t = tq * 8 + part;
                const float4 u0 = ld4(U0 + t * kVC + cg);
                const float4 u = make_float4(u0.x - a1[0], u0.y - a1[1], u0.z - a1[2], u0.w - a1[3]);
                *reinterpret_cast<float4*>(U + (item * kQ + t) * V + v0 + cg) = u;
                const float f = fs[c & 1][t];
                *reinterpret_cast<float4*>(Us + t * kLdU + cg) = make_float4(u.x * f, u.y * f, u.z * f, u.w * f);
            }
        } else {
            for (int i = tid; i < kQ * kVC / 4; i += kThreads) {
                const int t = i / (kVC / 4), e = (i % (kVC / 4)) * 4;
                const float f = fs[c & 1][t];
                const float4 u = ld4(U0 + t * kVC + e);
                *reinterpret_cast<float4*>(Us + t * kLdU + e) = make_float4(u.x * f, u.y * f, u.z * f, u.w * f);
            }
        }
        __syncthreads();
        {
            // rows of S: 4 dg .. + 3 and D / 2 + 4 dg .. + 3
            const int dg = (lane & 7) + 8 * (warp / 4), part = lane >> 3, cg = (warp & 3) * 4;
            float acc[8][4] = {};
#pragma unroll 4
            for (int t = part; t < kQ; t += 4) {
                const float4 x = ld4(Kc + t * D + 4 * dg), y = ld4(Kc + t * D + D / 2 + 4 * dg), u = ld4(Us + t * kLdU + cg);
                const float kv[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w}, uv[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(kv[i], uv[j], acc[i][j]);
            }
            // the four lanes' sums: after the two exchanges a lane holds one column's eight rows
            float a2[8][2], a1[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const bool up = part & 2;
                    const float keep = up ? acc[i][j + 2] : acc[i][j], give = up ? acc[i][j] : acc[i][j + 2];
                    a2[i][j] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
                }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const bool up = part & 1;
                const float keep = up ? a2[i][1] : a2[i][0], give = up ? a2[i][0] : a2[i][1];
                a1[i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
            }
            const float e = es[c & 1];
            float* s = St + (cg + part) * kLdS + 4 * dg;
            float4 x = ld4(s), y = ld4(s + D / 2);
            x = make_float4(fmaf(e, x.x, a1[0]), fmaf(e, x.y, a1[1]), fmaf(e, x.z, a1[2]), fmaf(e, x.w, a1[3]));
            y = make_float4(fmaf(e, y.x, a1[4]), fmaf(e, y.y, a1[5]), fmaf(e, y.z, a1[6]), fmaf(e, y.w, a1[7]));
            *reinterpret_cast<float4*>(s) = x;
            *reinterpret_cast<float4*>(s + D / 2) = y;
        }
        __syncthreads();  // the stage may be filled again
    }
    ns_pdl_launch_dependents();
    for (int i = tid; i < D * kVC; i += kThreads) S_mem[(size_t)(i / kVC) * V + i % kVC] = St[(i % kVC) * kLdS + i / kVC];
}

// ---------------------------------------------------------------------------------------
// grid (chunk slots, heads, V / VT), 256 threads: o = e Q S^T + M U with M = exp(L_t - L_s) (q_t . k_s), s <= t.  Warps of 32 tokens x VT / 4
// columns; S (transposed, its rows contiguous) comes in pieces of 64 of its rows, then U.
// ---------------------------------------------------------------------------------------
template <int D, int VT>
__global__ void __launch_bounds__(256, 2)
chunk_read_kernel(const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, const float* __restrict__ gate,
                  const float* __restrict__ decay, int ld, const int* __restrict__ qo_indptr, int n_requests, int min_len,
                  const float* __restrict__ U, const float* __restrict__ states, float* __restrict__ out, int ld_out, int H, int G, int V) {
    ns_pdl_wait();
    constexpr int kLdQ = D + 4, kLdS = 64 + 4, kLdU = VT + 4, kTN = VT / 32;
    constexpr int kX = kQ * kLdQ > VT * kLdS ? (kQ * kLdQ > kQ * kLdU ? kQ * kLdQ : kQ * kLdU) : (VT * kLdS > kQ * kLdU ? VT * kLdS : kQ * kLdU);
    extern __shared__ __align__(16) float read_smem[];
    float* Qs = read_smem;          // [64][D + 4]
    float* Xs = Qs + kQ * kLdQ;     // K [64][D + 4]; then S [VT][64 + 4], 64 of its rows at a time; then U [64][VT + 4]
    float* Ms = Xs + kX;            // [64][68]
    __shared__ double L[kQ];
    __shared__ Chunk chunk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, v0 = blockIdx.z * VT;
    if (warp == 0) {
        const Chunk c = find_chunk(blockIdx.x, qo_indptr, n_requests, min_len);
        if (lane == 0) chunk = c;
        if (c.count > 0) gate_logs(gate ? gate + h : nullptr, ld, decay ? decay[h] : 1.f, c.start, c.count, L);
    }
    __syncthreads();
    const Chunk c = chunk;
    if (c.count == 0) return;
    const size_t item = (size_t)c.slot * H + h, head = (size_t)(h / (H / G)) * D;
    stage<256, D>(Qs, kLdQ, q + (size_t)c.start * ld + head, ld, c.count);
    stage<256, D>(Xs, kLdQ, k + (size_t)c.start * ld + head, ld, c.count);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int ly = lane >> 3, lx = lane & 7;
    if (warp < 3) {  // a lower 32 x 32 block of Q K^T each
        const int tr = warp ? 32 : 0, sc = warp == 2 ? 32 : 0;
        float acc[8][4] = {};
        dot_rows<8, 4>(acc, Qs + (tr + ly) * kLdQ, kLdQ, Xs + (sc + lx) * kLdQ, kLdQ, D);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int t = tr + ly + 4 * i, s = sc + lx + 8 * j;
                Ms[t * kLdT + s] = s <= t ? expf((float)(L[t] - L[s])) * acc[i][j] : 0.f;
            }
    }
    const int tr = (warp >> 2) * 32, vc = (warp & 3) * (VT / 4);
    float y[8][kTN] = {};
    const float* Sg = states + (item * V + v0) * D;
    for (int d0 = 0; d0 < D; d0 += 64) {
        __syncthreads();
        for (int i = tid; i < VT * 16; i += 256) cp_async16(Xs + (i >> 4) * kLdS + (i & 15) * 4, Sg + (size_t)(i >> 4) * D + d0 + (i & 15) * 4, true);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        dot_rows<8, kTN>(y, Qs + (tr + ly) * kLdQ + d0, kLdQ, Xs + (vc + lx) * kLdS, kLdS, 64);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float f = expf((float)L[tr + ly + 4 * i]);
#pragma unroll
        for (int j = 0; j < kTN; ++j) y[i][j] *= f;
    }
    __syncthreads();
    if (U) stage<256, VT>(Xs, kLdU, U + item * kQ * V + v0, V, kQ);
    else stage<256, VT>(Xs, kLdU, v + (size_t)c.start * ld + (size_t)h * V + v0, ld, c.count);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    for (int s0 = 0; s0 < tr + 32; s0 += 32) {
        float run[8][kTN] = {};
        // tokens s0 + 4 m .. + 3; in the diagonal block a row t = ly + 4 i (counted from s0) ends at its own token
        auto add = [&](int m, bool diagonal) {
            float b[4][kTN];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int j = 0; j < kTN; ++j) b[u][j] = Xs[(s0 + 4 * m + u) * kLdU + vc + lx + 8 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (diagonal && i < m) continue;
                const float4 a = ld4(Ms + (tr + ly + 4 * i) * kLdT + s0 + 4 * m);
                const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (!diagonal || i > m || u <= ly) {
#pragma unroll
                        for (int j = 0; j < kTN; ++j) run[i][j] = fmaf(av[u], b[u][j], run[i][j]);
                    }
            }
        };
        if (s0 < tr) {
#pragma unroll 2
            for (int m = 0; m < 8; ++m) add(m, false);
        } else {
#pragma unroll
            for (int m = 0; m < 8; ++m) add(m, true);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < kTN; ++j) y[i][j] += run[i][j];
    }
    ns_pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = tr + ly + 4 * i;
        if (t >= c.count) continue;
        float* dst = out + (size_t)(c.start + t) * ld_out + (size_t)h * V + v0 + vc + lx;
#pragma unroll
        for (int j = 0; j < kTN; ++j) dst[8 * j] = y[i][j];
    }
}

template <int D, int VT>
int launch_read(const float* q, const float* k, const float* v, const float* gate, const float* decay, int ld, const int* qo_indptr, int n_requests,
                int min_len, const float* U, const float* states, float* out, int ld_out, int chunks, int H, int G, int V, cudaStream_t stream) {
    constexpr int kLdQ = D + 4;
    constexpr int x1 = kQ * kLdQ, x2 = VT * 68, x3 = kQ * (VT + 4), kX = x1 > x2 ? (x1 > x3 ? x1 : x3) : (x2 > x3 ? x2 : x3);
    constexpr size_t smem = sizeof(float) * (kQ * kLdQ + kX + kQ * kLdT);
    NS_CUDA(cudaFuncSetAttribute(chunk_read_kernel<D, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    NS_LAUNCH((chunk_read_kernel<D, VT>), dim3(chunks, H, V / VT), 256, smem, stream, q, k, v, gate, decay, ld, qo_indptr, n_requests, min_len, U, states,
              out, ld_out, H, G, V);
    NS_CHECK_LAUNCH("ns_linear_chunked");
    return NS_OK;
}

template <int D>
int launch_all(const float* q, const float* k, const float* v, const float* gate, const float* beta, const float* decay, int ld, float* state,
               long long state_floats, const int* qo_indptr, const int* state_slot, float* out, int ld_out, int n_requests, int min_len, int chunks,
               float* scratch, int H, int G, int V, cudaStream_t stream) {
    const bool delta = beta != nullptr;
    const size_t items = (size_t)chunks * H;
    float* states = scratch;
    float* fade = states + items * V * D;
    float* whole = fade + items * kQ;
    float* W = whole + (items + 3) / 4 * 4;
    float* U = W + items * kQ * D;
    constexpr size_t solve_smem = sizeof(float) * (kQ * (D + 4) + kQ * 132 + 2 * kQ * kLdT + 3 * 16 * 17);
    NS_CUDA(cudaFuncSetAttribute(chunk_solve_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)solve_smem));
    NS_LAUNCH((chunk_solve_kernel<D>), dim3(chunks, H), 256, solve_smem, stream, delta ? k : nullptr, v, gate, beta, decay, ld, qo_indptr, n_requests,
              min_len, W, U, fade, whole, H, G, V);
    NS_CHECK_LAUNCH("ns_linear_chunked");
    const dim3 walk(n_requests, H, V / kVC);
    constexpr size_t base = sizeof(float) * (kVC * (D + 4) + kQ * (kVC + 4));
    if (delta) {
        constexpr size_t smem = base + sizeof(float) * 2 * (2 * kQ * D + kQ * kVC);
        NS_CUDA(cudaFuncSetAttribute(chunk_walk_kernel<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        NS_LAUNCH((chunk_walk_kernel<D, true>), walk, 2 * D, smem, stream, k, v, ld, W, U, fade, whole, states, state, state_floats, qo_indptr, state_slot,
                  min_len, H, G, V);
    } else {
        constexpr size_t smem = base + sizeof(float) * 2 * (kQ * D + kQ * kVC);
        NS_CUDA(cudaFuncSetAttribute(chunk_walk_kernel<D, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        NS_LAUNCH((chunk_walk_kernel<D, false>), walk, 2 * D, smem, stream, k, v, ld, nullptr, nullptr, fade, whole, states, state, state_floats,
                  qo_indptr, state_slot, min_len, H, G, V);
    }
    NS_CHECK_LAUNCH("ns_linear_chunked");
    const float* u = delta ? U : nullptr;
    if (V % 128 == 0)
        return launch_read<D, 128>(q, k, v, gate, decay, ld, qo_indptr, n_requests, min_len, u, states, out, ld_out, chunks, H, G, V, stream);
    return launch_read<D, 64>(q, k, v, gate, decay, ld, qo_indptr, n_requests, min_len, u, states, out, ld_out, chunks, H, G, V, stream);
}

}  // namespace

// q, k, v, gate, beta: the columns of the preparation's rows (row stride ld floats), as ns_linear_scan takes them; beta null: retention, and
// gate null: `decay` per head.  Requests of fewer than min_len tokens are not touched; `chunks`: at least the chunks of the others.
// D 64 or 128, V a multiple of 64; `scratch`, on a 16-byte boundary: per chunk and head V * D + 65 floats, with beta 64 * (D + V) more, and 4.
NS_API int ns_linear_chunked(const float* q, const float* k, const float* v, const float* gate, const float* beta, const float* decay, int ld,
                             float* state, long long state_floats, const int* qo_indptr, const int* state_slot, float* out, int ld_out,
                             int n_requests, int min_len, int chunks, float* scratch, int H, int G, int D, int V, cudaStream_t stream) {
    if (n_requests <= 0 || chunks <= 0) return NS_OK;
    if (G < 1 || H % G) NS_FAIL(NS_ERR_ARGUMENT, "ns_linear_chunked: %d heads over %d key heads", H, G);
    if ((D != 64 && D != 128) || V < 64 || V % 64) NS_FAIL(NS_ERR_UNSUPPORTED, "ns_linear_chunked: a state of %d x %d", D, V);
    if (!gate && !decay) NS_FAIL(NS_ERR_ARGUMENT, "ns_linear_chunked: neither a gate per token nor a decay per head");
    if (ld % 4 || (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)scratch) % 16))
        NS_FAIL(NS_ERR_ARGUMENT, "ns_linear_chunked: rows of q, k and v and the scratch must start on 16 bytes");
    if (H > 65535 || V / kVC > 65535) NS_FAIL(NS_ERR_UNSUPPORTED, "ns_linear_chunked: %d heads of %d columns exceed the grid", H, V);
    if (D == 64)
        return launch_all<64>(q, k, v, gate, beta, decay, ld, state, state_floats, qo_indptr, state_slot, out, ld_out, n_requests, min_len, chunks,
                              scratch, H, G, V, stream);
    return launch_all<128>(q, k, v, gate, beta, decay, ld, state, state_floats, qo_indptr, state_slot, out, ld_out, n_requests, min_len, chunks, scratch,
                           H, G, V, stream);
}
