// The exact attention of csrc/attention_generic.cu for portions of prompts in float32: the same sums in the same order (the results
// agree bit for bit, so a position's output does not depend on whether its token came alone or in a portion), with the keys and
// values of a request read once per 32 query rows instead of once per row.
//
// A block takes a run of tokens of one request and one kv head: its rows are (token, query head of that kv head), 32 / (nq / nkv)
// tokens of them, eight rows to each of four warps.  Keys and values come 32 at a time through two cp.async stages.  A lane is a key in the
// scores (a chain of fmaf over the features in ascending order, as there) and a feature in the sums over the values (keys in
// ascending order, as there); a warp's eight rows share every read of a key or a value.
//
// Bound by the chain of a block's keys where few blocks share an SM (32 keys: 5,300 cycles, of them copies 650, scores 1,600, softmax 1,100, values 1,200), by
// shared memory (1,450 of its cycles for the same) where many do.  Three prompts of 300, 200 and 141 tokens, 32 heads of 64 over 8: 92 -> 55 us; one
// of 300 tokens, 4 heads over 1: 74 -> 32 us.  Of 11,000 cycles for 32 keys, 5,000 went into copies whose addresses shared registers, so that each
// waited for the data of the one before it, and 1,800 into the rows' reductions, one after the other.
#include "common.cuh"

namespace {

constexpr int kWarps = 4, kQ = 8, kRows = kWarps * kQ, kKeys = 32;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// DPL: features of a value per lane.  `tiles`: (request, offset among its tokens of this step) of runs of `tile_q` tokens.
template <int DPL>
__global__ void __launch_bounds__(kWarps * 32)
attention_f32_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                     const int* __restrict__ block_table, int table_stride, const int* __restrict__ positions,
                     const int* __restrict__ qo_indptr, const int* __restrict__ tiles, int tile_q, float* __restrict__ out, int o_stride,
                     int nq, int nkv, int d, int dv, int page_size, float scale, float softcap, const float* __restrict__ sink,
                     const float* __restrict__ gate, int gate_stride, int gate_per_feature, float out_scale) {
    ns_pdl_launch_dependents();
    ns_pdl_wait();
    extern __shared__ __align__(16) float f32_smem[];
    const int group = nq / nkv, tpb = kRows / group;
    const int req = tiles[2 * blockIdx.z], first = qo_indptr[req];
    const int len = qo_indptr[req + 1] - first;
    // (the later tokens of a run see the most keys and start first)
    const int off = tiles[2 * blockIdx.z + 1] + (int)(gridDim.x - 1 - blockIdx.x) * tpb;
    const int off_end = min(len, min(off + tpb, tiles[2 * blockIdx.z + 1] + tile_q));
    if (off >= off_end) return;
    const int n0 = first + off, rows = (off_end - off) * group;
    const int hk = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ldk = d + 4, pieces_k = d / 4, pieces_v = dv / 4;
    float* qs = f32_smem;                            // [kRows][d]
    float* ps = qs + kRows * d;                      // [kWarps][kKeys][kQ]
    float* ks = ps + kWarps * kKeys * kQ;            // [2][kKeys][d + 4]
    float* vs = ks + 2 * kKeys * ldk;                // [2][kKeys][dv]
    const int* bt = block_table + (size_t)req * table_stride;
    const int key_end = positions[first + off_end - 1] + 1;  // of the block's last token
    const int n_blocks = (key_end + kKeys - 1) / kKeys;

    // a lane's key of a block (beyond the end: the last one again, never used): where it is, found one block ahead of its copy
    auto find = [&](int kb) {
        const int key = min(kb * kKeys + lane, key_end - 1);
        return ((size_t)bt[key / page_size] * nkv + hk) * page_size + key % page_size;
    };
    size_t slot = find(0);
    auto issue = [&](int kb) {
        if (kb < n_blocks) {
            float* kd = ks + (kb & 1) * kKeys * ldk + warp * (kKeys / kWarps) * ldk;
            float* vd = vs + (kb & 1) * kKeys * dv + warp * (kKeys / kWarps) * dv;
            // straight code and an address register to each copy: copies whose addresses shared registers waited for one another's data
            const float *kg[kKeys / kWarps], *vg[kKeys / kWarps];
#pragma unroll
            for (int j = 0; j < kKeys / kWarps; ++j) {  // (a warp takes eight keys)
                const size_t at = __shfl_sync(0xffffffffu, slot, warp * (kKeys / kWarps) + j);
                kg[j] = k_cache + at * d + 4 * lane;
                vg[j] = v_cache + at * dv + 4 * lane;
            }
#pragma unroll
            for (int j = 0; j < kKeys / kWarps; ++j) {
                if (lane < pieces_k) cp_async16(kd + j * ldk + 4 * lane, kg[j]);
                if (lane + 32 < pieces_k) cp_async16(kd + j * ldk + 4 * lane + 128, kg[j] + 128);
                if (lane < pieces_v) cp_async16(vd + j * dv + 4 * lane, vg[j]);
                if (DPL > 4 && lane + 32 < pieces_v) cp_async16(vd + j * dv + 4 * lane + 128, vg[j] + 128);
            }
            slot = find(kb + 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);
    for (int i = tid; i < kRows * d; i += kWarps * 32) {
        const int r = i / d, e = i - r * d;
        qs[i] = r < rows ? q[(size_t)(n0 + r / group) * q_stride + (size_t)(hk * group + r % group) * d + e] : 0.f;
    }

    const int r0 = warp * kQ, mine = min(kQ, rows - r0);  // this warp's rows (none or fewer for the last warps of a short run)
    float m[kQ], l[kQ], acc[kQ][DPL];
    int kend[kQ], kend_min = 0x7fffffff, kend_max = 0;
#pragma unroll
    for (int i = 0; i < kQ; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
        kend[i] = i < mine ? positions[n0 + (r0 + i) / group] + 1 : 0;
        if (i < mine) { kend_min = min(kend_min, kend[i]); kend_max = max(kend_max, kend[i]); }
        else kend_min = 0;
#pragma unroll
        for (int u = 0; u < DPL; ++u) acc[i][u] = 0.f;
    }
    float* pw = ps + warp * kKeys * kQ;

    for (int kb = 0; kb < n_blocks; ++kb) {
        issue(kb + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();  // block kb (and at first the queries) are there for everybody
        if (kb * kKeys < kend_max) {
            const float* kr = ks + (kb & 1) * kKeys * ldk + lane * ldk;
            const float* vr = vs + (kb & 1) * kKeys * dv + lane;
            const float* qw = qs + r0 * d;
            float s[kQ];
#pragma unroll
            for (int i = 0; i < kQ; ++i) s[i] = 0.f;
#pragma unroll 4
            for (int e = 0; e < d; e += 4) {
                const float4 b = *reinterpret_cast<const float4*>(kr + e);
                float4 a[kQ];
#pragma unroll
                for (int i = 0; i < kQ; ++i) a[i] = *reinterpret_cast<const float4*>(qw + i * d + e);
#pragma unroll
                for (int i = 0; i < kQ; ++i) s[i] = fmaf(a[i].x, b.x, s[i]);
#pragma unroll
                for (int i = 0; i < kQ; ++i) s[i] = fmaf(a[i].y, b.y, s[i]);
#pragma unroll
                for (int i = 0; i < kQ; ++i) s[i] = fmaf(a[i].z, b.z, s[i]);
#pragma unroll
                for (int i = 0; i < kQ; ++i) s[i] = fmaf(a[i].w, b.w, s[i]);
            }
            // the eight rows' reductions side by side: one after the other they were most of the block's time
            const int key = kb * kKeys + lane;
            float top[kQ], corr[kQ];
#pragma unroll
            for (int i = 0; i < kQ; ++i) s[i] *= scale;
            if (softcap > 0.f) {
#pragma unroll
                for (int i = 0; i < kQ; ++i) s[i] = softcap * tanhf(s[i] / softcap);
            }
#pragma unroll
            for (int i = 0; i < kQ; ++i) top[i] = s[i] = key < kend[i] ? s[i] : -INFINITY;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < kQ; ++i) top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], o));
#pragma unroll
            for (int i = 0; i < kQ; ++i) {
                const float m_new = fmaxf(m[i], top[i]);
                corr[i] = expf(m[i] - m_new);  // (1 for a row that has seen all its keys)
                s[i] = expf(s[i] - m_new);
                m[i] = m_new;
                top[i] = s[i];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < kQ; ++i) top[i] += __shfl_xor_sync(0xffffffffu, top[i], o);
#pragma unroll
            for (int i = 0; i < kQ; ++i) {
                l[i] = l[i] * corr[i] + top[i];
#pragma unroll
                for (int u = 0; u < DPL; ++u) acc[i][u] *= corr[i];
            }
#pragma unroll
            for (int i = 0; i < kQ; i += 4) *reinterpret_cast<float4*>(pw + lane * kQ + i) = make_float4(s[i], s[i + 1], s[i + 2], s[i + 3]);
            __syncwarp();
            // blocks that every row sees whole, and the last ones, where a row's sums end at its last key (a value beyond it may be anything)
            auto add_values = [&](int j, bool all) {
                const float4 p0 = *reinterpret_cast<const float4*>(pw + j * kQ), p1 = *reinterpret_cast<const float4*>(pw + j * kQ + 4);
                const float p[kQ] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
                for (int u = 0; u < DPL; ++u) {
                    const float v = lane + 32 * u < dv ? vr[j * dv + 32 * u] : 0.f;
#pragma unroll
                    for (int i = 0; i < kQ; ++i)
                        if (all || kb * kKeys + j < kend[i]) acc[i][u] = fmaf(p[i], v, acc[i][u]);
                }
            };
            if (kb * kKeys + kKeys <= kend_min) {
#pragma unroll 8
                for (int j = 0; j < kKeys; ++j) add_values(j, true);
            } else {
                const int cnt = min(kKeys, kend_max - kb * kKeys);
#pragma unroll 4
                for (int j = 0; j < cnt; ++j) add_values(j, false);
            }
        }
        __syncthreads();  // the stage may be filled again
    }

#pragma unroll
    for (int i = 0; i < kQ; ++i) {
        if (i >= mine) break;
        const int n = n0 + (r0 + i) / group, h = hk * group + (r0 + i) % group;
        float li = l[i];
        if (sink) {  // a term of the denominator that has no key and no value: exp(sink[h])
            const float m_new = fmaxf(m[i], sink[h]);
            const float corr = expf(m[i] - m_new);
            li = li * corr + expf(sink[h] - m_new);
#pragma unroll
            for (int u = 0; u < DPL; ++u) acc[i][u] *= corr;
        }
        float inv = out_scale / li;
        if (gate && !gate_per_feature) inv *= 1.f / (1.f + expf(-gate[(size_t)n * gate_stride + h]));  // the head's output gate
        const float* fg = gate && gate_per_feature ? gate + (size_t)n * gate_stride + (size_t)h * dv : nullptr;  // ... or one per feature
        float* o = out + (size_t)n * o_stride + (size_t)h * dv;
#pragma unroll
        for (int u = 0; u < DPL; ++u) {
            const int e = lane + 32 * u;
            if (e < dv) o[e] = fg ? acc[i][u] * inv / (1.f + expf(-fg[e])) : acc[i][u] * inv;
        }
    }
}

size_t smem_bytes(int d, int dv) { return sizeof(float) * ((size_t)kRows * d + kWarps * kKeys * kQ + 2 * kKeys * (d + 4) + 2 * (size_t)kKeys * dv); }

template <int DPL, typename... Args>
int launch(dim3 grid, size_t smem, cudaStream_t stream, Args... args) {
    NS_CUDA(cudaFuncSetAttribute(attention_f32_kernel<DPL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    NS_LAUNCH((attention_f32_kernel<DPL>), grid, kWarps * 32, smem, stream, args...);
    NS_CHECK_LAUNCH("ns_attention_f32_tiles");
    return NS_OK;
}

}  // namespace

// tiles: int32 [n_tiles, 2] of (request, offset among its tokens of this step), runs of up to tile_q tokens; every key at or before a query's
// position is visible.  Head sizes in multiples of 4 up to 256, up to 32 query heads to a kv head.  `sink`, `gate`, `out_scale`: see
// ns_attention_generic_sink.
NS_API int ns_attention_f32_tiles(const float* q, int q_stride, const float* k_cache, const float* v_cache, const int* block_table,
                                  int table_stride, const int* positions, const int* qo_indptr, const int* tiles, int n_tiles, int tile_q,
                                  float* out, int o_stride, int nq, int nkv, int d, int dv, int page_size, float scale, float softcap,
                                  const float* sink, const float* gate, int gate_stride, int gate_per_feature, float out_scale,
                                  cudaStream_t stream) {
    if (n_tiles <= 0) return NS_OK;
    if (nkv < 1 || nq % nkv || nq / nkv > kRows) NS_FAIL(NS_ERR_UNSUPPORTED, "ns_attention_f32_tiles: %d query heads over %d kv heads", nq, nkv);
    if (d < 4 || d > 256 || d % 4 || dv < 4 || dv > 256 || dv % 4)
        NS_FAIL(NS_ERR_UNSUPPORTED, "ns_attention_f32_tiles: head sizes %d (keys) and %d (values) must be multiples of 4 up to 256", d, dv);
    if (((uintptr_t)k_cache | (uintptr_t)v_cache) % 16) NS_FAIL(NS_ERR_ARGUMENT, "ns_attention_f32_tiles: the cache must start on 16 bytes");
    if (tile_q < 1 || page_size < 1 || n_tiles > 65535 || nkv > 65535) NS_FAIL(NS_ERR_ARGUMENT, "ns_attention_f32_tiles: %d tiles of %d tokens, pages of %d", n_tiles, tile_q, page_size);
    const int tpb = kRows / (nq / nkv);
    const dim3 grid((tile_q + tpb - 1) / tpb, nkv, n_tiles);
    const size_t smem = smem_bytes(d, dv);
#define NS_F32_CASE(D)                                                                                                                       \
    case D:                                                                                                                                  \
        return launch<D>(grid, smem, stream, q, q_stride, k_cache, v_cache, block_table, table_stride, positions, qo_indptr, tiles, tile_q,  \
                         out, o_stride, nq, nkv, d, dv, page_size, scale, softcap, sink, gate, gate_stride, gate_per_feature, out_scale);
    switch ((dv + 31) / 32) { NS_F32_CASE(1) NS_F32_CASE(2) NS_F32_CASE(3) NS_F32_CASE(4) NS_F32_CASE(5) NS_F32_CASE(6) NS_F32_CASE(7) NS_F32_CASE(8) }
#undef NS_F32_CASE
    NS_FAIL(NS_ERR_UNSUPPORTED, "ns_attention_f32_tiles: values of %d", dv);
}
