// 32-bit matrix product on the 5th-generation tensor cores: y[M, N] = x[M, K] * w[N, K]^T, nothing rounded to less than 24 bits.
//
// Floats come apart into three bfloat16, exactly, a product of two into six products (csrc/float_parts.cuh).  The tensor core multiplies parts exactly and
// adds them in float32, but it truncates, so its chains are kept short and small things go first: in every block of 64 k the five
// products with a middle or a low part, then the four steps of high by high, into an accumulator that starts at zero; the block's sum
// then joins its group's sum in registers, rounded to nearest, and the groups (eight at most, of at least 512 k, by K alone) are added in their order.
//
// An element's value depends on its row of x, its row of w and K: the order of its sums is the same for every M, every tile and every split, so
// rows alone and in a batch give the same bits.  Parts are 2^24 times the floats, so that small ones keep all their bits; an infinity or a NaN among
// them, numbers from 2^104 and sums from 2^80 on come out infinite or NaN, and such an element is formed again from the floats themselves by
// its warp (32 chains of fmaf and their sum).
//
// The product is computed transposed, as in gemm_tcgen05.cu: 128 rows of w are the M side of tcgen05.mma, bn rows of x (16 to 96) its N side.
// A block owns an SM and walks over tiles (blockIdx.x, + gridDim.x, ...; the tiles of the same rows of w are neighbours, so that w comes from DRAM
// once); where there are fewer tiles than SMs, a cluster of blocks shares a tile's groups and adds them up through distributed shared memory.
// Warp roles, in this order:
//   1    loads w: floats into a ring of shared memory, by TMA
//   1    issues the MMAs
//   1    loads x's parts by TMA (f32_parts_kernel has taken x apart once, since every tile of w would do it again)
//   1    waits for all that a block's MMAs need
//   8    take w's tile apart and write its parts to TMEM as the A operand (a thread owns a row): shared memory then serves the tensor core with
//        x alone
//   4-12 add a finished block's accumulator to their sums in registers (32 columns to a thread), add up groups, write results
//
// Weights that a checkpoint held in 16 bits have neither middle nor low parts.  Where a block's 128 x 64 of w have none, the three products with
// them are left out: they are zeros, so the bits stay (641 x 16384 x 2048 213 -> 163 us).  The eight warps see the parts as they make them.
//
// Microseconds on a B200 in a graph of such products (w from DRAM): the kernels of gemm_f32.cu, this one with its parts kernel on weights of 24 bits,
// and on bfloat16's numbers
//     M x N x K   1 x 2048 x 2048   8 x 2048 x 8192   3 x 32768 x 2048   200 x 8192 x 1024   641 x 2048 x 8192   641 x 16384 x 2048   8 x 1024 x 512
//     fmaf               23                97                 89                 119                 709                 943                 7.0
//     24 bits            11.0              25                 51                  30                 120                 213                 9.0
//     bfloat16's         10.8              24                 50                  27                  92                 163                 9.0
// From K = 1024 on the GPU was slower nowhere (1 x 1024 x 1024: 11.6 / 10.5); that line is the dispatch's (F32_TC_MIN_K).  The host is: an eager product
// of a few rows takes it 15 us, two launches and the parts' buffer, where one launch took 9.  Groups that were added up in y
// (a read-modify-write of the tile for each) took 244 us instead of 213 on 641 x 16384 x 2048, 128 instead of 117 on 641 x 2048 x 8192.
// Error against 64 bits (2-norm, normal x and w), one chain of fmaf / this kernel, in 1e-7: K = 1024 5.7 / 1.0, 2048 8.1 / 1.0, 8192 16 / 1.2,
// 14336 21 / 1.4; numbers over 60 powers of two 7.0 / 1.3; all of one sign 6.3 / 0.9.  Rows of x with few numbers that are not zero are the other way
// round, since a chain of n fmaf rounds n times: with one 0.25 / 0.46, 4 0.41 / 0.59, 8 0.54 / 0.66, 16 0.74 / 0.72, 128 2.0 / 0.9.
// Elements formed from the floats cost what they are: 641 x 16384 x 2048 with an infinity in every row 13 ms, with a NaN in every row (found once for
// 32 elements) 0.75.
// Bound, with 96 rows, by shared memory, which the MMAs' operand, TMA's writes and the reads of w share (24 bits: 1,700 cycles a block of k, of which
// the MMAs run for 1,190; bfloat16's numbers: 1,290 and 600); with 16 rows (990 cycles) by taking w apart.
//
// The accumulators are double buffered, both operands' parts have three or four stages (a warpgroup of the eight warps takes every other block),
// so that taking apart, multiplying and adding up do not wait for one another.
#include <cfloat>
#include <type_traits>

#include "float_parts.cuh"
#include "tcgen05_utils.cuh"

namespace {

constexpr int kBM = 128, kBK = 64, kMaxBN = 96;
constexpr int kRingBytes = kBM * kBK * 4;        // a stage of floats of w: two boxes of 128 rows x 32 floats
constexpr int kMaxRing = 6, kMaxStages = 4;      // stages of w's ring and of the parts at most
constexpr int kSmemMax = 227 * 1024;
constexpr int kBarBytes = 384, kSmemFixed = 1024 + kBarBytes;  // barriers; alignment
constexpr uint32_t kTmemCols = 512;              // two accumulators, then the stages of w's parts (32 columns to a part)
constexpr uint32_t kPartsCols = kParts * kBK / 2;

enum F32TcError { kErrF32Loader = 51, kErrF32Mma = 52, kErrF32Weights = 53, kErrF32Rows = 54, kErrF32Sum = 55, kErrF32Drain = 56 };

// Elements from the floats themselves: a lane whose `mine` is set gets the product of x and row `lane` of w.  Four rows of w at a time; a NaN in x is
// the result of them all, found in one reading of it.  Apart from the kernel's code, whose registers are counted.
__device__ __noinline__ float warp_dots(const float* __restrict__ x, const float* __restrict__ w, int ldw, int K, bool mine) {
    const int lane = threadIdx.x & 31;
    unsigned who = __ballot_sync(0xffffffffu, mine);
    bool nan = false;
    for (int k = lane; k < K; k += 32) nan |= x[k] != x[k];
    if (__any_sync(0xffffffffu, nan)) return __int_as_float(0x7fffffff);
    float result = 0.f;
    int last = 0;
    while (who) {
        int src[4];
        float p[4];
        const float* row[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // (fewer than four left: the last one again)
            if (who) last = __ffs(who) - 1;
            src[i] = last;
            who &= who - 1;
            row[i] = w + (size_t)src[i] * ldw;
            p[i] = 0.f;
        }
#pragma unroll 4
        for (int k = lane; k < K; k += 32) {
            const float v = x[k];
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = fmaf(v, row[i][k], p[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            p[i] = ns_warp_sum(p[i]);
            if (lane == src[i]) result = p[i];
        }
    }
    return result;
}

struct F32Gemm {
    const float* x;
    const float* w;
    float* y;
    int M, N, K, ldx, ldw, ldy;
    int bn, m_tiles, tiles, k_blocks, group_blocks, groups;
    int ring;  // stages of w's ring
};

__device__ __forceinline__ bool out_of_range(float v) { return !(fabsf(v) <= FLT_MAX); }
// a warp's 32 results of row m (rows n_warp + lane of w), which it has written: those that the parts cannot give come from the floats
__device__ __forceinline__ void mend_row(const F32Gemm& a, int m, int n_warp) {
    const int lane = threadIdx.x & 31;
    float* out = a.y + (size_t)m * a.ldy + n_warp + lane;
    const bool odd = n_warp + lane < a.N && out_of_range(*out);
    if (!__any_sync(0xffffffffu, odd)) return;
    const float p = warp_dots(a.x + (size_t)m * a.ldx, a.w + (size_t)n_warp * a.ldw, a.ldw, a.K, odd);
    if (odd) *out = p;
}

// tiles of up to kBN rows of x: the roles' first warps, stages of both operands' parts
template <int kBN>
struct Roles {
    static constexpr int kW = 4, kSum = kW + 8, kSumWarps = kBN / 32 * 4, kThreads = 32 * (kSum + kSumWarps);
    static constexpr int kStages = kBN <= 32 ? 4 : 3;
    static constexpr uint32_t kXPart = kBN * 128, kXStage = kParts * kXPart;  // bytes, whatever bn is
    static_assert(2 * kBN + kStages * kPartsCols <= kTmemCols, "tensor memory");
};

// x[M, K] -> parts[3][M][ldp]: high, middle, low; eight k to a thread, zeros from K to ldp
__global__ void __launch_bounds__(256) f32_parts_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ parts, int M, int K, int ldx, int ldp, int pieces) {
    ns_pdl_wait();
    ns_pdl_launch_dependents();  // in this order: the product loads w without a wait of its own, and a kernel before this one may have written it
    const int per_row = ldp / 8;
    const size_t plane = (size_t)M * ldp;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < (long long)M * per_row; i += (long long)gridDim.x * 256) {
        const int m = (int)(i / per_row), k = (int)(i - (long long)m * per_row) * 8;
        const float* src = x + (size_t)m * ldx + k;
        float v[8];
        if (pieces && k + 8 <= K) {
            ld8(src, v);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = k + j < K ? src[j] : 0.f;
        }
        uint32_t p[kParts][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split_pair(v[2 * j], v[2 * j + 1], p[0][j], p[1][j], p[2][j]);
#pragma unroll
        for (int q = 0; q < kParts; ++q) *reinterpret_cast<uint4*>(parts + q * plane + (size_t)m * ldp + k) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
}

template <int kBN>
__global__ void __launch_bounds__(Roles<kBN>::kThreads, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const F32Gemm a, int splits,
                   int* __restrict__ error_flag) {
    using R = Roles<kBN>;
    extern __shared__ unsigned char smem_dyn[];
    const uint32_t base = (smem_u32(smem_dyn) + 1023u) & ~1023u;
    constexpr uint32_t part_bytes = R::kXPart;
    constexpr int stages = R::kStages;
    const int bn = a.bn, ring = a.ring;
    const uint32_t x_smem = base, w_smem = base + stages * R::kXStage;
    const uint32_t bar0 = w_smem + (uint32_t)ring * kRingBytes;
    auto w_full = [&](int s) { return bar0 + 8u * s; };
    auto w_empty = [&](int s) { return bar0 + 8u * (kMaxRing + s); };
    auto x_full = [&](int s) { return bar0 + 8u * (2 * kMaxRing + s); };
    auto w_ready = [&](int s) { return bar0 + 8u * (2 * kMaxRing + kMaxStages + s); };    // w's parts are in TMEM
    auto empty = [&](int s) { return bar0 + 8u * (2 * kMaxRing + 2 * kMaxStages + s); };  // the MMAs that read a stage of parts are complete,
    constexpr int kRings = 2 * kMaxRing + 3 * kMaxStages;
    auto done = [&](int b) { return bar0 + 8u * (kRings + b); };                            // and so is the accumulator
    auto acc_free = [&](int b) { return bar0 + 8u * (kRings + 2 + b); };                    // which has been read
    auto go = [&](int s) { return bar0 + 8u * (kRings + 4 + s); };                          // all that a block's MMAs wait for is there
    const uint32_t holder = bar0 + 8u * (kRings + 4 + kMaxStages);
    auto finer = [&](int s) { return bar0 + 8u * (kRings + 6 + kMaxStages) + 16u * s; };    // four warps' words: does w's tile have middle or low parts?
    static_assert(8 * (kRings + 6 + kMaxStages) % 16 == 0 && 8 * (kRings + 6 + kMaxStages) + 16 * kMaxStages <= kBarBytes, "barriers");
    float* groups_smem = reinterpret_cast<float*>(smem_dyn + (bar0 + (uint32_t)kBarBytes - smem_u32(smem_dyn)));  // splits > 1: this block's groups [group][row of x][128]
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (known to be one number for the warp)

    if (threadIdx.x == 0) {
        for (int s = 0; s < ring; ++s) {
            mbar_init(w_full(s), 1);
            mbar_init(w_empty(s), 4);
        }
        for (int s = 0; s < stages; ++s) {
            mbar_init(x_full(s), 1);
            mbar_init(w_ready(s), 4);
            mbar_init(empty(s), 1);
            mbar_init(go(s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(done(b), 1);
            mbar_init(acc_free(b), R::kSumWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_smem();
    }
    if (warp == 1) tmem_alloc(holder, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    uint32_t tmem_base;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(tmem_base) : "r"(holder));
    tmem_base = __shfl_sync(0xffffffffu, tmem_base, 0);

    // what this block does: tiles first, first + step, ...; blocks [kb0, kb0 + n_kb) of each; g counts them in every role
    const int rank = (int)blockIdx.x % splits, first = (int)blockIdx.x / splits, step = (int)gridDim.x / splits;
    const int per_rank = (a.groups + splits - 1) / splits;
    const int kb0 = min(rank * per_rank * a.group_blocks, a.k_blocks), n_kb = min((rank + 1) * per_rank * a.group_blocks, a.k_blocks) - kb0;
    const int my_tiles = first < a.tiles ? (a.tiles - 1 - first) / step + 1 : 0;
    const int total = my_tiles * n_kb;
    auto tile_at = [&](int i, int& m0, int& n0) {
        const int t = first + i * step, n = t / a.m_tiles;
        n0 = n * kBM;
        m0 = (t - n * a.m_tiles) * bn;
    };

    if (warp == 0) {
        // ---------------- w's floats: the predecessor, f32_parts_kernel, does not write them and has waited for all before it ----------------
        int g = 0;
        bool ok = true;
        for (int i = 0; ok && i < my_tiles; ++i) {
            int m0, n0;
            tile_at(i, m0, n0);
            for (int kb = kb0; kb < kb0 + n_kb; ++kb, ++g) {
                const int s = g % ring;
                if (g >= ring && !mbar_wait_warp(w_empty(s), (uint32_t)(g / ring - 1) & 1u)) {
                    ok = false;
                    if (lane == 0) atomicExch(error_flag, kErrF32Loader);
                    break;
                }
                if (elect_one()) {
                    mbar_expect_tx(w_full(s), kRingBytes);
                    const uint32_t dst = w_smem + (uint32_t)s * kRingBytes;
                    tma_load_2d(dst, &map_w, kb * kBK, n0, w_full(s));
                    tma_load_2d(dst + kRingBytes / 2, &map_w, kb * kBK + 32, n0, w_full(s));
                }
            }
        }
        for (int i = max(0, g - ring); i < g; ++i)  // nothing may still be landing when the block leaves
            if (!mbar_wait_warp(w_full(i % ring), (uint32_t)(i / ring) & 1u)) {
                if (lane == 0) atomicExch(error_flag, kErrF32Drain);
                break;
            }
    } else if (warp == 1) {
        // ---------------- MMAs ----------------
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
        int s = 0, issued = 0;
        uint32_t s_turn = 0;
        for (int g = 0; g < total; ++g) {
            const int b = g & 1;
            if (!mbar_wait_warp(go(s), s_turn)) {
                if (lane == 0) atomicExch(error_flag, kErrF32Mma);
                break;
            }
            tc_fence_after();
            const uint32_t d = tmem_base + (uint32_t)b * kBN, wp = tmem_base + 2 * kBN + (uint32_t)s * kPartsCols;
            const uint64_t xp = smem_desc(x_smem + (uint32_t)s * R::kXStage);
            // Weights that bfloat16 holds exactly (a checkpoint of that type run in float32) have no middle or low parts: three of the six products
            // are zeros, and adding zeros changes nothing.
            uint32_t f[4];
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3]) : "r"(finer(s)) : "memory");
            // Unrolled, a lane elected for each, offsets known to the compiler: operands that are not in uniform registers cost an MMA more to
            // issue than it runs (it runs for 20 cycles with 16 columns, 55 with 96; issued from a branch of one lane it took 126).
            auto products = [&](auto with_parts_of_w) {
                constexpr bool kAll = decltype(with_parts_of_w)::value;
                constexpr int pw[6] = {2, 0, 1, 1, 0, 0}, px[6] = {0, 2, 1, 0, 1, 0};
                bool first = true;
#pragma unroll
                for (int p = 0; p < 6; ++p) {
                    if (!kAll && pw[p] != 0) continue;
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k) {
                        if (elect_one())
                            umma_bf16_ts(d, wp + pw[p] * 32 + k * 8, xp + ((px[p] * part_bytes + k * 32) >> 4), idesc, first ? 0u : 1u);
                        first = false;
                    }
                }
            };
            if (__any_sync(0xffffffffu, (f[0] | f[1] | f[2] | f[3]) != 0)) products(std::true_type{});
            else products(std::false_type{});
            if (elect_one()) umma_commit(done(b));
            if (elect_one()) umma_commit(empty(s));
            if (++s == stages) { s = 0; s_turn ^= 1u; }
            ++issued;
        }
        for (int g = max(0, issued - stages); g < issued; ++g)  // nothing may still be multiplied, or arrive at a barrier, when the block leaves
            if (!mbar_wait_warp(empty(g % stages), (uint32_t)(g / stages) & 1u)) {
                if (lane == 0) atomicExch(error_flag, kErrF32Drain);
                break;
            }
    } else if (warp == 3) {
        // ---------------- waits for the MMAs: three barriers, 200 cycles each even when they are complete (shared memory is busy), would be the
        // issuer's own time otherwise (96 rows of x: 1,790 cycles a block of k) ----------------
        for (int g = 0; g < total; ++g) {
            const int s = g % stages, b = g & 1;
            const uint32_t s_turn = (uint32_t)(g / stages) & 1u;
            if (!mbar_wait_warp(x_full(s), s_turn) || !mbar_wait_warp(w_ready(s), s_turn) ||
                (g > 1 && !mbar_wait_warp(acc_free(b), ((uint32_t)(g >> 1) - 1u) & 1u))) {
                if (lane == 0) atomicExch(error_flag, kErrF32Mma);
                break;
            }
            tc_fence_after();
            tc_fence_before();
            if (lane == 0) mbar_arrive(go(s));
        }
    } else if (warp == 2) {
        // ---------------- x's parts, as f32_parts_kernel left them ----------------
        ns_pdl_wait();
        int g = 0;
        bool ok = true;
        for (int i = 0; ok && i < my_tiles; ++i) {
            int m0, n0;
            tile_at(i, m0, n0);
            for (int kb = kb0; kb < kb0 + n_kb; ++kb, ++g) {
                const int s = g % stages;
                if (g >= stages && !mbar_wait_warp(empty(s), (uint32_t)(g / stages - 1) & 1u)) {
                    ok = false;
                    if (lane == 0) atomicExch(error_flag, kErrF32Rows);
                    break;
                }
                if (elect_one()) {
                    mbar_expect_tx(x_full(s), kParts * (uint32_t)bn * 128u);
                    const uint32_t dst = x_smem + (uint32_t)s * kParts * part_bytes;
#pragma unroll
                    for (int q = 0; q < kParts; ++q)  // (rows beyond M are another part's or zeros: multiplied and not stored)
                        tma_load_2d(dst + q * part_bytes, &map_x, kb * kBK, q * a.M + m0, x_full(s));
                }
            }
        }
        for (int i = max(0, g - stages); i < g; ++i)
            if (!mbar_wait_warp(x_full(i % stages), (uint32_t)(i / stages) & 1u)) {
                if (lane == 0) atomicExch(error_flag, kErrF32Drain);
                break;
            }
    } else if (warp < R::kSum) {
        // ---------------- w's parts: a thread owns a row ----------------
        const int quarter = warp & 3;
        const uint32_t row_off = (uint32_t)(quarter * 32 + lane) * 128u, sw = (uint32_t)(lane & 7);
        const uint32_t t_row = tmem_base + 2 * kBN + ((uint32_t)(quarter * 32) << 16);
        for (int g = (warp - R::kW) >> 2; g < total; g += 2) {
            const int s = g % ring, p = g % stages;
            // The parts' stage first: when it is free, w's tile `stages` blocks back has been read, so the ring's barrier cannot lie two phases back,
            // where its parity would say "full" (a stage of an odd ring goes from one warpgroup to the other; see launch_f32_tc).
            if ((g >= stages && !mbar_wait_warp(empty(p), (uint32_t)(g / stages - 1) & 1u)) || !mbar_wait_warp(w_full(s), (uint32_t)(g / ring) & 1u)) {
                if (lane == 0) atomicExch(error_flag, kErrF32Weights);
                break;
            }
            tc_fence_after();
            const uint32_t src = w_smem + (uint32_t)s * kRingBytes + row_off;
            uint32_t rest = 0;
            float4 v[2][4];  // 16 k at a time, the next ones on their way (read and taken apart in turn: 1,900 cycles a tile, most of them waiting)
            auto read = [&](int q) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                 : "=f"(v[q & 1][c].x), "=f"(v[q & 1][c].y), "=f"(v[q & 1][c].z), "=f"(v[q & 1][c].w)
                                 : "r"(src + (q >> 1) * (kRingBytes / 2) + (((uint32_t)((q & 1) * 4 + c) ^ sw) << 4)));
            };
            read(0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (q < 3) read(q + 1);
                uint32_t hi[8], mid[8], lo[8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    split_pair(v[q & 1][c].x, v[q & 1][c].y, hi[2 * c], mid[2 * c], lo[2 * c]);
                    split_pair(v[q & 1][c].z, v[q & 1][c].w, hi[2 * c + 1], mid[2 * c + 1], lo[2 * c + 1]);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) rest |= mid[c];  // (no middle part: no low one)
                if (q == 3) {
                    const bool any = __any_sync(0xffffffffu, (rest & 0x7fff7fffu) != 0);  // (a zero's sign is nothing)
                    if (lane == 0) {
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(finer(p) + 4u * quarter), "r"((int)any) : "memory");
                        mbar_arrive(w_empty(s));
                    }
                    __syncwarp();
                }
                const uint32_t dst = t_row + (uint32_t)p * kPartsCols + q * 8;
                tmem_st8(dst, hi);
                tmem_st8(dst + 32, mid);
                tmem_st8(dst + 64, lo);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(w_ready(p));
        }
    } else {
        // ---------------- sums: a thread owns a row of w and all or half of the tile's rows of x ----------------
        ns_pdl_wait();
        const int quarter = warp & 3, c0 = (warp - R::kSum) / 4 * 32, cols = min(32, bn - c0);  // (none left: the warp only keeps step)
        constexpr int kLoad = kBN <= 32 ? 32 : 8;  // columns at a time: 64 sums leave no more registers
        const uint32_t t_acc = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
        int g = 0;
        bool ok = true;
        for (int i = 0; ok && i < my_tiles; ++i) {
            int m0, n0;
            tile_at(i, m0, n0);
            const int n_warp = n0 + quarter * 32, n = n_warp + lane;
            float all[32];  // the groups so far
            for (int kb = kb0; kb < kb0 + n_kb;) {
                float sum[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) sum[j] = 0.f;
                const int group = kb / a.group_blocks, end = min((group + 1) * a.group_blocks, a.k_blocks);
                for (; kb < end; ++kb, ++g) {
                    const int b = g & 1;
                    if (!mbar_wait_warp(done(b), (uint32_t)(g >> 1) & 1u)) {
                        ok = false;
                        if (lane == 0) atomicExch(error_flag, kErrF32Sum);
                        break;
                    }
                    tc_fence_after();
                    if (cols > 0) {  // (columns past the tile's hold what other tiles left: added and not stored)
#pragma unroll
                        for (int c = 0; c < 32; c += kLoad) {
                            uint32_t r[kLoad];
                            if constexpr (kLoad == 8) tmem_ld8(t_acc + (uint32_t)b * kBN + c, r);
                            else tmem_ld32(t_acc + (uint32_t)b * kBN + c, r);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < kLoad; ++j) sum[c + j] += __uint_as_float(r[j]);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_free(b));
                }
                if (!ok) break;
                if (splits > 1) {
                    float* dst = groups_smem + (size_t)((group - rank * per_rank) * bn + c0) * kBM + quarter * 32 + lane;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (j < cols) dst[j * kBM] = sum[j];
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) all[j] = group == 0 ? sum[j] : all[j] + sum[j];
                }
            }
            if (!ok) break;
            if (splits > 1) continue;
            const int rows = n < a.N ? min(cols, a.M - m0 - c0) : 0;
            bool odd = false;
            float* out = a.y + (size_t)(m0 + c0) * a.ldy + n;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (j < rows) {
                    *out = all[j] * kPartsBack;
                    odd |= out_of_range(all[j]);
                }
                out += a.ldy;
                asm volatile("" : "+l"(out));  // (a running pointer: 32 addresses kept through the sums would not leave them their registers)
            }
            if (__any_sync(0xffffffffu, odd)) {
#pragma unroll 1
                for (int m = m0 + c0; m < min(m0 + c0 + cols, a.M); ++m) mend_row(a, m, n_warp);
            }
        }
    }
    __syncwarp();
    ns_pdl_wait();  // (every thread: see ns_launch_impl)
    if (splits > 1) {
        cluster_sync();  // every block's groups are in its shared memory
        const int rows = (bn + splits - 1) / splits, r0 = rank * rows, r1 = min(bn, r0 + rows);
        int m0, n0;
        tile_at(0, m0, n0);
        const uint32_t mine = smem_u32(groups_smem);
        for (int e = threadIdx.x >> 5; e < (r1 - r0) * 4; e += R::kThreads / 32) {  // 32 rows of w of a row of x to a warp
            const int r = r0 + (e >> 2), at = (e & 3) * 32 + lane, m = m0 + r, n_warp = n0 + (e & 3) * 32;
            if (m >= a.M) break;
            float v = 0.f;
            for (int q = 0; q < a.groups; ++q) {
                const float p = ld_cluster_f32(mine + (uint32_t)(((q % per_rank) * bn + r) * kBM + at) * 4u, (uint32_t)(q / per_rank));
                v = q == 0 ? p : v + p;
            }
            if (n_warp + lane < a.N) a.y[(size_t)m * a.ldy + n_warp + lane] = v * kPartsBack;
            if (__any_sync(0xffffffffu, out_of_range(v))) mend_row(a, m, n_warp);
        }
        cluster_sync();  // nobody leaves while its shared memory is read
    }
    tc_fence_before();
    __syncthreads();
    ns_pdl_launch_dependents();  // (not at once: a successor placed while this grid holds the SMs lands unevenly, see gemm_f32.cu)
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

template <int kBN>
int launch_f32_tc(const CUtensorMap& mw, const CUtensorMap& mx, F32Gemm a, int splits, int grid, int* error_flag, cudaStream_t stream) {
    using R = Roles<kBN>;
    const int held = splits > 1 ? (a.groups + splits - 1) / splits * a.bn * kBM * 4 : 0, fixed = kSmemFixed + held + R::kStages * (int)R::kXStage;
    a.ring = min(kMaxRing, (kSmemMax - fixed) / kRingBytes);
    if (a.ring % 2 && a.ring < R::kStages) --a.ring;  // (an odd ring is no shorter than the parts' stages, an even one keeps a stage to one warpgroup)
    if (a.ring < 2) NS_FAIL(NS_ERR_ARGUMENT, "ns_gemm_f32_tc: %d groups of %d rows in %d splits do not fit shared memory", a.groups, a.bn, splits);
    NS_CUDA(cudaFuncSetAttribute(gemm_f32_tc_kernel<kBN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(R::kThreads);
    cfg.dynamicSmemBytes = (size_t)(fixed + a.ring * kRingBytes);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (splits > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = splits;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (ns_take_pdl()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    NS_CUDA(cudaLaunchKernelEx(&cfg, gemm_f32_tc_kernel<kBN>, mw, mx, a, splits, error_flag));
    return NS_OK;
}

}  // namespace

// x: [M, K] with row stride ldx; w: [N, K] with row stride ldw, on 16 bytes with rows of 16-byte pieces (ldw and K multiples of 4); y: [M, N] with
// row stride ldy; parts: bfloat16 [3, M, K rounded up to 8], scratch; bn: rows of x to a tile, a multiple of 16
// up to 96; splits: 1, 2, 4 or 8 blocks to a tile (more than 1: no more tiles than n_sms / splits); n_sms: multiprocessors of the device;
// error_flag: a device int that a timed-out wait sets.
NS_API int ns_gemm_f32_tc(const float* x, const float* w, float* y, void* parts, int M, int N, int K, int ldx, int ldw, int ldy, int bn, int splits,
                          int n_sms, int* error_flag, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return NS_OK;
    if (K <= 0 || K % 4 || ldw % 4 || (uintptr_t)w % 16)
        NS_FAIL(NS_ERR_UNSUPPORTED, "ns_gemm_f32_tc: K=%d, rows of w %d apart: multiples of 4 on 16 bytes are wanted", K, ldw);
    if (bn < 16 || bn > kMaxBN || bn % 16) NS_FAIL(NS_ERR_ARGUMENT, "ns_gemm_f32_tc: tiles of %d rows", bn);
    const int ldp = (K + 7) / 8 * 8;
    if (!parts || (uintptr_t)parts % 16 || 3ll * M > 0x7fffffff) NS_FAIL(NS_ERR_ARGUMENT, "ns_gemm_f32_tc: no scratch for the parts of %d rows", M);
    const int k_blocks = (K + kBK - 1) / kBK, most = min(8, (k_blocks + 7) / 8), group_blocks = (k_blocks + most - 1) / most;
    const int groups = (k_blocks + group_blocks - 1) / group_blocks;
    const long long m_tiles = (M + bn - 1) / bn, tiles = (N + kBM - 1) / kBM * m_tiles;
    if (tiles > 0x7fffffff || (tiles / n_sms + 1) * k_blocks > 0x7fffffff) NS_FAIL(NS_ERR_UNSUPPORTED, "ns_gemm_f32_tc: %d x %d x %d has too many tiles", M, N, K);
    if (splits != 1 && splits != 2 && splits != 4 && splits != 8) NS_FAIL(NS_ERR_ARGUMENT, "ns_gemm_f32_tc: %d blocks to a tile", splits);
    if (splits > 1 && (splits > groups || tiles * splits > n_sms)) NS_FAIL(NS_ERR_ARGUMENT, "ns_gemm_f32_tc: %lld tiles of %d groups in %d splits", tiles, groups, splits);
    CUtensorMap mw, mx;
    if (const int rc = ns_make_map<4>(&mw, w, (unsigned long long)N, K, ldw, kBM, "ns_gemm_f32_tc")) return rc;
    if (const int rc = ns_make_map<2>(&mx, parts, 3ull * M, ldp, ldp, bn, "ns_gemm_f32_tc")) return rc;
    const long long blocks = ((long long)M * (ldp / 8) + 255) / 256;
    NS_LAUNCH(f32_parts_kernel, (unsigned)min(blocks, 8ll * n_sms), 256, 0, stream, x, (__nv_bfloat16*)parts, M, K, ldx, ldp,
              (int)(ldx % 4 == 0 && (uintptr_t)x % 16 == 0));
    NS_CHECK_LAUNCH("ns_gemm_f32_tc");
    const F32Gemm a = {x, w, y, M, N, K, ldx, ldw, ldy, bn, (int)m_tiles, (int)tiles, k_blocks, group_blocks, groups, 0};
    const int grid = splits > 1 ? (int)tiles * splits : (int)(tiles < n_sms ? tiles : n_sms);
    auto* launch = bn <= 32 ? launch_f32_tc<32> : launch_f32_tc<96>;
    return launch(mw, mx, a, splits, grid, error_flag, stream);
}
