// True 32-bit matrix product on the CUDA cores: y[M, N] = x[M, K] * w[N, K]^T.  Products of K below 1,024, and those whose w TMA cannot
// address; the others run in gemm_f32_tc.cu.
//
// No tensor cores and no reduced-precision mode: every product and sum is an fp32 FMA.
// Each output element is accumulated by one thread over k = 0..K-1 in ascending order, so
// its value does not depend on M, on the tile it falls in, or on what else is in the batch
// (the three kernels below give the same bits).  Rows that do not start on 16 bytes, and K that is no multiple of 4, run in the wide tiles.
//
// Microseconds on a B200, one 64 x 64 kernel with 4 x 4 results a thread before -> now (an FMA loop in registers reaches 72 TFLOP/s here):
//     M x N x K         3 x 32768 x 2048   8 x 2048 x 2048   128 x 2048 x 2048   641 x 2048 x 2048   641 x 2048 x 8192   641 x 16384 x 2048
//     before / now          352 / 89           145 / 26          150 / 70            337 / 179           1341 / 704         1441 / 1020
//
// The kernels start their successor when their sums are done and not at once: a successor of a few blocks an SM that is placed
// while this grid still holds most slots lands unevenly and then runs as long as its fullest SM (64 x 16384 x 2048 back to
// back: 206 us with the early start, 139 with the late one).
#include "common.cuh"

namespace {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// four consecutive k of a row, zeros beyond the matrix
template <bool kAligned>
__device__ __forceinline__ float4 load_k4(const float* __restrict__ base, int row, int rows, int ld, int k, int K) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows) {
        const float* p = base + (size_t)row * ld + k;
        if (kAligned && k + 3 < K) return *reinterpret_cast<const float4*>(p);
        if (k < K) v.x = p[0];
        if (k + 1 < K) v.y = p[1];
        if (k + 2 < K) v.z = p[2];
        if (k + 3 < K) v.w = p[3];
    }
    return v;
}

constexpr int BK = 16;

// ---------------------------------------------------------------------------------------
// Grids of a few blocks an SM: tiles of 32 x 64, two warps of 32 x 32, 8 x 4 results a thread.  Tiles lie in shared memory as in
// memory (k contiguous, rows 20 floats apart: the eight rows of a load's phase fall into different banks), four stages by cp.async; a thread
// reads four k of a row at a time.  Bound by what shared memory can return (12 words to 32 FMAs a thread), 57 % of the FMA
// rate; larger tiles lose more to the last wave than they win there (641 x 2048 x 2048: 32 x 64 179 us, 64 x 64 219, 64 x 128 266).
// ---------------------------------------------------------------------------------------
constexpr int kBM = 32, kBN = 64, kTM = 8, kTN = 4, kStages = 4, kLd = BK + 4, kTileThreads = 64;

__global__ void __launch_bounds__(kTileThreads)  // rows start on 16 bytes and K is a multiple of 4
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K,
                int ldx, int ldw, int ldy) {
    ns_pdl_wait();  // everything below sees the previous kernel's results
    constexpr int kStage = (kBM + kBN) * kLd;
    __shared__ __align__(16) float smem[kStages * kStage];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * kBM, n0 = blockIdx.x * kBN;
    const int r = lane >> 3, c = warp * 8 * kTN + (lane & 7);  // rows r, r + 4, ...; columns c, c + 8, ...
    const int n_tiles = (K + BK - 1) / BK;
    auto issue = [&](int t) {
        if (t < n_tiles) {
            float* st = smem + (t % kStages) * kStage;
#pragma unroll
            for (int p = tid; p < (kBM + kBN) * 4; p += kTileThreads) {
                const int row = p >> 2, k = t * BK + (p & 3) * 4;
                const bool is_x = row < kBM;
                const int g = is_x ? m0 + row : n0 + row - kBM;
                const bool in = g < (is_x ? M : N) && k < K;
                const float* src = is_x ? x + (size_t)g * ldx + k : w + (size_t)g * ldw + k;
                cp_async16(st + row * kLd + (p & 3) * 4, in ? src : w, in ? 16 : 0);
            }
        }
        cp_async_commit();
    };
    float acc[kTM][kTN];
#pragma unroll
    for (int i = 0; i < kTM; ++i)
#pragma unroll
        for (int j = 0; j < kTN; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int t = 0; t < kStages - 1; ++t) issue(t);
    for (int t = 0; t < n_tiles; ++t) {
        cp_async_wait<kStages - 2>();
        __syncthreads();  // tile t is there for everybody, and the stage of tile t - 1 has been read
        issue(t + kStages - 1);
        const float* xt = smem + (t % kStages) * kStage + r * kLd;
        const float* wt = smem + (t % kStages) * kStage + (kBM + c) * kLd;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 b[kTN];
#pragma unroll
            for (int j = 0; j < kTN; ++j) b[j] = *reinterpret_cast<const float4*>(wt + 8 * j * kLd + k);
#pragma unroll
            for (int i = 0; i < kTM; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(xt + 4 * i * kLd + k);
#pragma unroll
                for (int j = 0; j < kTN; ++j) acc[i][j] = fmaf(a.x, b[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < kTN; ++j) acc[i][j] = fmaf(a.y, b[j].y, acc[i][j]);
#pragma unroll
                for (int j = 0; j < kTN; ++j) acc[i][j] = fmaf(a.z, b[j].z, acc[i][j]);
#pragma unroll
                for (int j = 0; j < kTN; ++j) acc[i][j] = fmaf(a.w, b[j].w, acc[i][j]);
            }
        }
    }
    ns_pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < kTM; ++i) {
        const int gm = m0 + r + 4 * i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < kTN; ++j) {
            const int gn = n0 + c + 8 * j;
            if (gn < N) y[(size_t)gm * ldy + gn] = acc[i][j];
        }
    }
}

// ---------------------------------------------------------------------------------------
// Grids of many blocks: tiles of 64 x 128, four warps of 32 x 64, 8 x 8 results a thread as packed FMAs (fma.rn.f32x2: two fp32 FMAs
// to an issue slot, each rounded as fmaf rounds).  16 words of shared memory to 64 FMAs a thread, in tiles laid down transposed
// through registers one k tile ahead; two stages.  48 TFLOP/s at 2048 x 4096 x 4096 (1432 us; the kernel above 1616).
// ---------------------------------------------------------------------------------------
constexpr int kWideM = 64, kWideN = 128, kWideThreads = 128;

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

template <bool kAligned>
__global__ void __launch_bounds__(kWideThreads, 3)
gemm_f32_wide_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K,
                     int ldx, int ldw, int ldy) {
    ns_pdl_wait();
    constexpr int kLdX = kWideM + 4, kLdW = kWideN + 4;
    constexpr int kPx = kWideM * BK / 4 / kWideThreads, kPw = kWideN * BK / 4 / kWideThreads;  // 16-byte pieces a thread stages
    __shared__ __align__(16) float xs[2][BK * kLdX];
    __shared__ __align__(16) float ws[2][BK * kLdW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * kWideM, n0 = blockIdx.x * kWideN;
    // a thread's rows r .. r + 3 and r + 16 .. r + 19, columns c .. c + 3 and c + 32 .. c + 35
    const int r = (warp >> 1) * 32 + (lane >> 3) * 4, c = (warp & 1) * 64 + (lane & 7) * 4;

    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;

    float4 px[kPx], pw[kPw];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < kPx; ++i) {
            const int p = tid + i * kWideThreads;
            px[i] = load_k4<kAligned>(x, m0 + (p >> 2), M, ldx, k0 + (p & 3) * 4, K);
        }
#pragma unroll
        for (int i = 0; i < kPw; ++i) {
            const int p = tid + i * kWideThreads;
            pw[i] = load_k4<kAligned>(w, n0 + (p >> 2), N, ldw, k0 + (p & 3) * 4, K);
        }
    };
    auto store = [&](int st) {
#pragma unroll
        for (int i = 0; i < kPx; ++i) {
            const int p = tid + i * kWideThreads;
            float* d = xs[st] + (p & 3) * 4 * kLdX + (p >> 2);
            d[0] = px[i].x; d[kLdX] = px[i].y; d[2 * kLdX] = px[i].z; d[3 * kLdX] = px[i].w;
        }
#pragma unroll
        for (int i = 0; i < kPw; ++i) {
            const int p = tid + i * kWideThreads;
            float* d = ws[st] + (p & 3) * 4 * kLdW + (p >> 2);
            d[0] = pw[i].x; d[kLdW] = pw[i].y; d[2 * kLdW] = pw[i].z; d[3 * kLdW] = pw[i].w;
        }
    };

    fetch(0);
    store(0);
    __syncthreads();
    const int n_tiles = (K + BK - 1) / BK;
    for (int t = 0; t < n_tiles; ++t) {
        const bool more = t + 1 < n_tiles;
        if (more) fetch((t + 1) * BK);
        const float* xt = xs[t & 1] + r;
        const float* wt = ws[t & 1] + c;
        // the operands of the next k are read while this one's products run
        float4 a[2][2];
        ulonglong2 b[2][2];
        auto read = [&](int k) {
            a[k & 1][0] = *reinterpret_cast<const float4*>(xt + k * kLdX);
            a[k & 1][1] = *reinterpret_cast<const float4*>(xt + k * kLdX + 16);
            b[k & 1][0] = *reinterpret_cast<const ulonglong2*>(wt + k * kLdW);
            b[k & 1][1] = *reinterpret_cast<const ulonglong2*>(wt + k * kLdW + 32);
        };
        read(0);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            if (k + 1 < BK) read(k + 1);
            const float4 a0 = a[k & 1][0], a1 = a[k & 1][1];
            const ulonglong2 b0 = b[k & 1][0], b1 = b[k & 1][1];
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t aa = pack2(av[i], av[i]);
                fma2(acc[i][0], aa, b0.x);
                fma2(acc[i][1], aa, b0.y);
                fma2(acc[i][2], aa, b1.x);
                fma2(acc[i][3], aa, b1.y);
            }
        }
        if (more) store((t + 1) & 1);  // (the stage was last read before the barrier at the end of the tile before)
        __syncthreads();
    }
    ns_pdl_launch_dependents();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gm = m0 + r + (i < 4 ? i : 12 + i);
        if (gm >= M) continue;
        float* row = y + (size_t)gm * ldy;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 v = unpack2(acc[i][j]);
            const int gn = n0 + c + (j < 2 ? 2 * j : 28 + 2 * j);
            if (gn < N) row[gn] = v.x;
            if (gn + 1 < N) row[gn + 1] = v.y;
        }
    }
}

// ---------------------------------------------------------------------------------------
// A few rows: the weights are what such a product moves.  A block takes 32 columns (a lane each) and all rows, R to each of
// its four warps; tiles of 64 k come through four cp.async stages, a lane reads its column's weights four k at a time and the rows of
// x as broadcasts.  3 x 32768 x 2048: 3.0 TB/s.
// ---------------------------------------------------------------------------------------
constexpr int kRowsK = 64, kRowsLd = kRowsK + 4;

template <int R>
__global__ void __launch_bounds__(128)
gemm_f32_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K, int ldx, int ldw, int ldy) {
    ns_pdl_launch_dependents();  // (short: the next kernel may as well be scheduled now)
    ns_pdl_wait();
    extern __shared__ __align__(16) float rows_smem[];
    constexpr int kRows = 32 + 4 * R, kStage = kRows * kRowsLd;  // 32 rows of w, then the rows of x
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * 32;
    const int n_tiles = (K + kRowsK - 1) / kRowsK;
    auto issue = [&](int t) {
        if (t < n_tiles) {
            float* st = rows_smem + (t % kStages) * kStage;
            for (int p = tid; p < kRows * (kRowsK / 4); p += 128) {
                const int row = p / (kRowsK / 4), k = t * kRowsK + (p % (kRowsK / 4)) * 4;
                const bool is_w = row < 32;
                const int g = is_w ? n0 + row : row - 32;
                const bool in = (is_w ? g < N : g < M) && k < K;  // (K is a multiple of 4: a piece is in or out; what is out reads as zeros)
                const float* src = is_w ? w + (size_t)g * ldw + k : x + (size_t)g * ldx + k;
                cp_async16(st + row * kRowsLd + (p % (kRowsK / 4)) * 4, in ? src : w, in ? 16 : 0);
            }
        }
        cp_async_commit();
    };
    float acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.f;
#pragma unroll
    for (int t = 0; t < kStages - 1; ++t) issue(t);
    for (int t = 0; t < n_tiles; ++t) {
        cp_async_wait<kStages - 2>();
        __syncthreads();  // tile t is there for everybody, and the stage of tile t - 1 has been read
        issue(t + kStages - 1);
        const float* st = rows_smem + (t % kStages) * kStage;
        const float* wr = st + lane * kRowsLd;
        const float* xr = st + (32 + warp * R) * kRowsLd;
#pragma unroll
        for (int k = 0; k < kRowsK; k += 4) {
            const float4 b = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const float4 a = *reinterpret_cast<const float4*>(xr + i * kRowsLd + k);
                acc[i] = fmaf(a.x, b.x, acc[i]);
                acc[i] = fmaf(a.y, b.y, acc[i]);
                acc[i] = fmaf(a.z, b.z, acc[i]);
                acc[i] = fmaf(a.w, b.w, acc[i]);
            }
        }
    }
    const int n = n0 + lane;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (warp * R + i < M && n < N) y[(size_t)(warp * R + i) * ldy + n] = acc[i];
}

template <int R>
int launch_rows(const float* x, const float* w, float* y, int M, int N, int K, int ldx, int ldw, int ldy, cudaStream_t stream) {
    constexpr size_t bytes = sizeof(float) * kStages * (32 + 4 * R) * kRowsLd;
    NS_CUDA(cudaFuncSetAttribute(gemm_f32_rows_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    NS_LAUNCH((gemm_f32_rows_kernel<R>), (N + 31) / 32, 128, bytes, stream, x, w, y, M, N, K, ldx, ldw, ldy);
    NS_CHECK_LAUNCH("ns_gemm_f32");
    return NS_OK;
}

}  // namespace

// x: [M, K] with row stride ldx; w: [N, K] with row stride ldw; y: [M, N] with row stride ldy; n_sms: multiprocessors of the device.
NS_API int ns_gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, int ldx, int ldw, int ldy,
                       int n_sms, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return NS_OK;
    if (K <= 0) NS_FAIL(NS_ERR_ARGUMENT, "ns_gemm_f32: K=%d", K);
    if ((M + 63) / 64 > 65535) NS_FAIL(NS_ERR_UNSUPPORTED, "ns_gemm_f32: M=%d exceeds 65535 row tiles", M);
    const bool aligned = (ldx % 4 == 0) && (ldw % 4 == 0) && (((uintptr_t)x | (uintptr_t)w) % 16 == 0);
    // up to 16 rows, and up to 32 where the columns alone would not give every SM a tile (32 x 2048 x 8192: 169 us against about 280 in
    // tiles; 32 x 16384 x 2048: 133 against about 75)
    if (aligned && K % 4 == 0 && (M <= 16 || (M <= 32 && N <= (long long)kBN * n_sms))) {
        if (M <= 4) return launch_rows<1>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
        if (M <= 8) return launch_rows<2>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
        if (M <= 16) return launch_rows<4>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
        return launch_rows<8>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
    }
    // Wide tiles from six blocks an SM on (below that the last round costs more than it wins: 641 x 3072 x 2048
    // 236 against 233 us, 641 x 2048 x 2048 235 against 179), with more rows than the small tiles' grid can hold, and whenever the small
    // tiles' 16-byte copies cannot be had: their loads go through registers a tile ahead (rows of 2,049, 16 x 2048 124 us, 300 x 2048
    // 129, 1500 x 2048 314; small tiles filled by plain loads 190, 261, 632).
    const dim3 wide((N + kWideN - 1) / kWideN, (M + kWideM - 1) / kWideM), small((N + kBN - 1) / kBN, (M + kBM - 1) / kBM);
    const bool pieces = aligned && K % 4 == 0;
    if (!pieces || (long long)wide.x * wide.y >= 6LL * n_sms || small.y > 65535) {
        if (aligned) NS_LAUNCH((gemm_f32_wide_kernel<true>), wide, kWideThreads, 0, stream, x, w, y, M, N, K, ldx, ldw, ldy);
        else NS_LAUNCH((gemm_f32_wide_kernel<false>), wide, kWideThreads, 0, stream, x, w, y, M, N, K, ldx, ldw, ldy);
    } else {
        NS_LAUNCH(gemm_f32_kernel, small, kTileThreads, 0, stream, x, w, y, M, N, K, ldx, ldw, ldy);
    }
    NS_CHECK_LAUNCH("ns_gemm_f32");
    return NS_OK;
}
