// KV-cache append (RoPE + f32->f16) and split-KV flash-decode attention with GQA, head_dim 128.
//
// Layouts follow the reference everywhere: q/out f32 [head][128]; K/V f16 [pos][kv_head][128]
// (crates/rnb-cpu/src/kernels/attention/decode_flash.rs:13-15,
//  crates/rnb-backend/cuda/cuda/kernels/gdn_attention.cuh:1733-1734).
// Decode attention is a pure KV stream: each K/V row is read from HBM once per KV group and
// shared by the `group` query heads that map to it; all arithmetic is fp32.
#pragma once
#include "common.cuh"
#include "q8k.cuh"

namespace rnb {

constexpr int HD = 128;

// RoPE on q and k with a host-built cos/sin table row (the reference's fused path also builds
// its tables on the host: crates/rnb-backend/cuda/src/runtime/state/rope_cache.rs:33-54; the
// values here come from the CPU angle chain of crates/rnb-cpu/src/kernels/rope.rs:267-293),
// then K/V rows are rounded to f16 (round-to-nearest-even, as half::f16::from_f32 in
// crates/rnb-llm/src/kv_cache.rs:126-141) and written at row `pos` of the layer's cache.
// grid = num_heads + 2*num_kv_heads CTAs of 64 threads; thread i owns rotation pair i.
// rope_table: [max_pos][2][64] (cos then sin) indexed by position when table_by_pos != 0,
// else a single row.  Position = *pos_dev (optional device scalar) + pos_offset.
RNB_GLOBAL void __launch_bounds__(64)
rope_kv_append_kernel(float *q, const float *k,
                      const float *v, const float *__restrict__ rope_table,
                      const int *pos_dev, int pos_offset, int table_by_pos,
                      int num_heads, int num_kv_heads, int neox, uint16_t *k_cache,
                      uint16_t *v_cache, uint16_t *k_row_out,
                      uint16_t *v_row_out) {
    pdl_launch_dependents();
    pdl_wait();
    // gridDim.y > 1: a batch of consecutive tokens (prefill), token t = blockIdx.y at position base + t,
    // its q/k/v rows t * (heads or kv heads) * 128 further on
    q += (size_t)blockIdx.y * num_heads * HD;
    k += (size_t)blockIdx.y * num_kv_heads * HD;
    v += (size_t)blockIdx.y * num_kv_heads * HD;
    const int pos = (pos_dev ? *pos_dev : 0) + pos_offset + (int)blockIdx.y;
    const int i = threadIdx.x;
    const float *cs = rope_table + (size_t)(table_by_pos ? pos : 0) * 128;
    const float c = cs[i], s = cs[64 + i];
    const int i0 = neox ? i : 2 * i, i1 = neox ? i + 64 : 2 * i + 1;
    int h = blockIdx.x;
    if (h < num_heads) {
        float *qh = q + (size_t)h * HD;
        const float x0 = qh[i0], x1 = qh[i1];
        qh[i0] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
        qh[i1] = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
        return;
    }
    h -= num_heads;
    const size_t kv_dim = (size_t)num_kv_heads * HD;
    if (h < num_kv_heads) {
        const float *kh = k + (size_t)h * HD;
        const float x0 = kh[i0], x1 = kh[i1];
        const uint16_t r0 = __half_as_ushort(__float2half_rn(__fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s))));
        const uint16_t r1 = __half_as_ushort(__float2half_rn(__fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c))));
        if (k_cache) {
            uint16_t *dst = k_cache + (size_t)pos * kv_dim + (size_t)h * HD;
            dst[i0] = r0;
            dst[i1] = r1;
        }
        if (k_row_out) {
            k_row_out[(size_t)h * HD + i0] = r0;
            k_row_out[(size_t)h * HD + i1] = r1;
        }
        return;
    }
    h -= num_kv_heads;
    const float *vh = v + (size_t)h * HD;
    const uint16_t r0 = __half_as_ushort(__float2half_rn(vh[i])),
                   r1 = __half_as_ushort(__float2half_rn(vh[i + 64]));
    if (v_cache) {
        uint16_t *dst = v_cache + (size_t)pos * kv_dim + (size_t)h * HD;
        dst[i] = r0;
        dst[i + 64] = r1;
    }
    if (v_row_out) {
        v_row_out[(size_t)h * HD + i] = r0;
        v_row_out[(size_t)h * HD + i + 64] = r1;
    }
}

// The same work for a batch of consecutive tokens (prefill): one CTA of 256 threads per token,
// thread (g = tid / 64, i = tid % 64) owns rotation pair i of heads g, g + 4, ... - the cos/sin of
// the pair is read once.  Same arithmetic and rounding as rope_kv_append_kernel.
RNB_GLOBAL void __launch_bounds__(256)
rope_kv_append_tokens_kernel(float *q, const float *k, const float *v, const float *__restrict__ rope_table,
                             int pos0, int num_heads, int num_kv_heads, int neox, uint16_t *k_cache, uint16_t *v_cache) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, pos = pos0 + t, i = threadIdx.x & 63, g = threadIdx.x >> 6;
    const float *cs = rope_table + (size_t)pos * 128;
    const float c = cs[i], s = cs[64 + i];
    const int i0 = neox ? i : 2 * i, i1 = neox ? i + 64 : 2 * i + 1;
    const size_t kv_dim = (size_t)num_kv_heads * HD;
    float *qt = q + (size_t)t * num_heads * HD;
    for (int h = g; h < num_heads; h += 4) {
        float *qh = qt + (size_t)h * HD;
        const float x0 = qh[i0], x1 = qh[i1];
        qh[i0] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
        qh[i1] = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
    }
    const float *kt = k + (size_t)t * kv_dim, *vt = v + (size_t)t * kv_dim;
    uint16_t *kd = k_cache + (size_t)pos * kv_dim, *vd = v_cache + (size_t)pos * kv_dim;
    for (int h = g; h < num_kv_heads; h += 4) {
        const float *kh = kt + (size_t)h * HD;
        const float x0 = kh[i0], x1 = kh[i1];
        kd[(size_t)h * HD + i0] = __half_as_ushort(__float2half_rn(__fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s))));
        kd[(size_t)h * HD + i1] = __half_as_ushort(__float2half_rn(__fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c))));
    }
    for (size_t e = threadIdx.x; e < kv_dim; e += 256) vd[e] = __half_as_ushort(__float2half_rn(vt[e]));
}

// Plain f32 -> f16 row append (no RoPE) for callers that rotate elsewhere.
RNB_GLOBAL void kv_append_f16_kernel(const float *src, uint16_t *dst,
                                     size_t n) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = __half_as_ushort(__float2half_rn(src[i]));
}

// ---- split-KV flash decode ------------------------------------------------------------------
// grid = (num_kv_heads, n_chunks); 128 threads.  Chunk c covers positions
// [c*chunk_len, min(kv_len, (c+1)*chunk_len)) with chunk_len = ceil(kv_len / n_chunks) rounded
// up to 8.  Warp w walks positions c0+w, c0+w+4, ...; lane l owns dims 4l..4l+3 of the row.
// Per (head, chunk) the kernel writes an un-normalised accumulator, the running max and the
// running sum into `partials` ([num_heads][n_chunks][HD + 2] floats); flash_decode_reduce
// merges chunks with the usual log-sum-exp rule.
constexpr int FD_THREADS = 128;
constexpr int FD_PART_STRIDE = HD + 2;
constexpr int FD_MAX_CHUNKS = 1024;   // merge kernels keep one rescale factor per chunk in shared memory

// four consecutive K/V elements as f32, from an f16 cache (decode) or f32 tensors (prefill API)
__device__ __forceinline__ float4 kv_load4(const uint16_t *p) {
    const uint2 b = *reinterpret_cast<const uint2 *>(p);
    const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&b.x));
    const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&b.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ float4 kv_load4(const float *p) {
    return *reinterpret_cast<const float4 *>(p);
}

// G = query heads handled per pass (<= group size).  When `direct_out` is given the merged,
// normalised result is written there ([head][128]) instead of a partial record.
template <int G, typename KVT>
__device__ __forceinline__ void fd_process(const float *q, const KVT *k,
                                           const KVT *v, int kv_h, int head0,
                                           int heads_here, size_t kv_dim, int p_begin, int p_end,
                                           float scale, int n_chunks, int chunk,
                                           float *partials, float *s_acc, float *s_ml,
                                           float *direct_out = nullptr) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float qr[G][4], acc[G][4], m[G], l[G];
#pragma unroll
    for (int g = 0; g < G; g++) {
        const float4 qv = g < heads_here
                              ? *reinterpret_cast<const float4 *>(q + (size_t)(head0 + g) * HD + 4 * lane)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
        qr[g][0] = qv.x * scale;
        qr[g][1] = qv.y * scale;
        qr[g][2] = qv.z * scale;
        qr[g][3] = qv.w * scale;
        acc[g][0] = acc[g][1] = acc[g][2] = acc[g][3] = 0.f;
        m[g] = -INFINITY;
        l[g] = 0.f;
    }
    const size_t head_off = (size_t)kv_h * HD + 4 * lane;
#pragma unroll 2
    for (int p = p_begin + warp; p < p_end; p += FD_THREADS / 32) {
        const float4 kk = kv_load4(k + (size_t)p * kv_dim + head_off);
        const float4 vv = kv_load4(v + (size_t)p * kv_dim + head_off);
        float sc[G];
#pragma unroll
        for (int g = 0; g < G; g++)
            sc[g] = qr[g][0] * kk.x + qr[g][1] * kk.y + qr[g][2] * kk.z + qr[g][3] * kk.w;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int g = 0; g < G; g++) sc[g] += __shfl_xor_sync(0xffffffffu, sc[g], o);
#pragma unroll
        for (int g = 0; g < G; g++) {
            const float mn = fmaxf(m[g], sc[g]);
            const float corr = expf(m[g] - mn);  // m = -inf on the first position -> 0
            const float pw = expf(sc[g] - mn);
            acc[g][0] = acc[g][0] * corr + pw * vv.x;
            acc[g][1] = acc[g][1] * corr + pw * vv.y;
            acc[g][2] = acc[g][2] * corr + pw * vv.z;
            acc[g][3] = acc[g][3] * corr + pw * vv.w;
            l[g] = l[g] * corr + pw;
            m[g] = mn;
        }
    }
    // merge the 4 warps' states through shared memory
    __syncthreads();
#pragma unroll
    for (int g = 0; g < G; g++) {
        float *a = s_acc + ((size_t)(warp * G + g)) * HD + 4 * lane;
        a[0] = acc[g][0];
        a[1] = acc[g][1];
        a[2] = acc[g][2];
        a[3] = acc[g][3];
        if (lane == 0) {
            s_ml[(warp * G + g) * 2] = m[g];
            s_ml[(warp * G + g) * 2 + 1] = l[g];
        }
    }
    __syncthreads();
    for (int g = 0; g < heads_here; g++) {
        const int d = threadIdx.x;  // 128 threads <-> 128 dims
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < FD_THREADS / 32; w++) M = fmaxf(M, s_ml[(w * G + g) * 2]);
        float a = 0.f, L = 0.f;
#pragma unroll
        for (int w = 0; w < FD_THREADS / 32; w++) {
            const float mw = s_ml[(w * G + g) * 2];
            const float f = mw == -INFINITY ? 0.f : expf(mw - M);
            a += s_acc[((size_t)(w * G + g)) * HD + d] * f;
            L += s_ml[(w * G + g) * 2 + 1] * f;
        }
        if (direct_out) {
            direct_out[(size_t)(head0 + g) * HD + d] = L > 0.f ? a / L : 0.f;
            continue;
        }
        float *out = partials + ((size_t)(head0 + g) * n_chunks + chunk) * FD_PART_STRIDE;
        out[d] = a;
        if (d == 0) {
            out[HD] = M;
            out[HD + 1] = L;
        }
    }
}

RNB_GLOBAL void __launch_bounds__(FD_THREADS)
flash_decode_partials_kernel(const float *q, const uint16_t *k,
                             const uint16_t *v, const int *kv_len_dev,
                             int kv_len_host, int num_heads, int num_kv_heads, float scale,
                             float *partials) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float s_acc[(FD_THREADS / 32) * 4 * HD];
    __shared__ float s_ml[(FD_THREADS / 32) * 4 * 2];
    const int kv_len = kv_len_dev ? *kv_len_dev + kv_len_host : kv_len_host;
    const int n_chunks = gridDim.y, chunk = blockIdx.y, kv_h = blockIdx.x;
    int chunk_len = (kv_len + n_chunks - 1) / n_chunks;
    chunk_len = (chunk_len + 7) & ~7;
    const int p_begin = min(kv_len, chunk * chunk_len), p_end = min(kv_len, p_begin + chunk_len);
    const int group = num_heads / num_kv_heads;
    const size_t kv_dim = (size_t)num_kv_heads * HD;
    for (int g0 = 0; g0 < group; g0 += 4) {
        const int here = min(4, group - g0);
        fd_process<4, uint16_t>(q, k, v, kv_h, kv_h * group + g0, here, kv_dim, p_begin, p_end,
                                scale, n_chunks, chunk, partials, s_acc, s_ml);
        __syncthreads();
    }
}

// ---- split-KV flash decode on the tensor cores (f16 caches) ---------------------------------
// Same grid, chunking and partial-record format as flash_decode_partials_kernel, but the K/V
// rows of a chunk are staged in shared memory by 256-byte bulk copies (one per row, completing
// on an mbarrier per 16-position block) and both products run as m16n8k16 MMAs with fp32
// accumulators, with the (up to 8) query heads of a KV group as the N dimension:
//   S^T[pos][head] = K[pos][dim] . Q^T[dim][head]     A = K rows as stored, B = query
//   O^T[dim][head] += V^T[dim][pos] . P^T[pos][head]  A = V rows read transposed, B = P
// K and V are exact f16 values; the pre-scaled f32 query and the f32 probabilities are each
// split into two f16 terms (hi + lo), so the products keep ~22 mantissa bits.
// Warp w owns positions [16w, 16w+16) of each 64-position staging pass and keeps its own
// running (max, sum, O); the four warps are merged through shared memory at the end.
constexpr int FDM_THREADS = 128;
constexpr int FDM_SUPER = 64;             // positions staged per pass
constexpr int FDM_ROW = 2 * HD + 16;      // padded row: ldmatrix without bank conflicts
constexpr int FDM_KV_BYTES = 2 * FDM_SUPER * FDM_ROW;
constexpr int FDM_ACC_STRIDE = HD + 4;    // merge scratch row (floats), padded against conflicts

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
__device__ __forceinline__ void mma_f16_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (x, y) -> f16x2 "hi" and the f16x2 remainder "lo"
__device__ __forceinline__ void split_f16x2(float x, float y, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(x, y);
    const float2 hf = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - hf.x, y - hf.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

// PREFILL = false: decode, grid (kv heads, chunks), one query, partial records out.
// PREFILL = true: causal prefill, grid (kv heads, query blocks); the 8 MMA columns are
// (8 / group) consecutive queries x the group's heads, query i sees positions
// 0 .. kv_len - seq_len + i, and the normalised result is written straight to `out`
// ([seq][head][128]); no chunking, the CTA walks all visible positions.
// Optional tail of the decode kernel: the CTA that completes a KV head's last chunk (arrival counter,
// re-armed by that CTA) merges the chunks of the group's query heads and writes the attention
// output as f32 and / or as Q8_K blocks (two heads = one 256-element block), which saves the merge
// launch.  counters: one int per KV head, zero before the launch.
struct FdMerge {
    int *counters;       // null: no counter-based merge
    float *out;          // [heads][128] f32, optional
    uint8_t *xq_out;     // Q8K-dev layout of the heads x 128 vector, optional (needs an even head group)
    int cluster;         // > 0: the launch is one thread-block cluster of this many chunks per KV head; the
                         // cluster's CTA b merges heads 2b, 2b + 1 of the group after a cluster barrier
};
template <bool PREFILL>
__device__ __forceinline__ void fdm_body(const float *q, const uint16_t *k, const uint16_t *v,
                                         const int *kv_len_dev, int kv_len_host, int seq_len, int num_heads, int num_kv_heads,
                                         float scale, float *partials, float *out, int *err_flag,
                                         const FdMerge merge = FdMerge{nullptr, nullptr, nullptr, 0}) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ __align__(128) uint8_t s_kv[FDM_KV_BYTES];   // K rows then V rows; merge scratch later
    __shared__ __align__(8) uint64_t s_bar[FDM_SUPER / 16];
    __shared__ float s_ml[(FDM_THREADS / 32) * 8 * 2], s_factor[(FDM_THREADS / 32) * 8], s_max[8];
    static_assert((FDM_THREADS / 32) * 8 * FDM_ACC_STRIDE * 4 <= FDM_KV_BYTES, "merge scratch must fit the staging area");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int kv_len = kv_len_dev ? *kv_len_dev + kv_len_host : kv_len_host;
    const int n_chunks = gridDim.y, chunk = blockIdx.y, kv_h = blockIdx.x;
    const int group = num_heads / num_kv_heads;
    const int qpc = PREFILL ? (group >= 8 ? 1 : 8 / group) : 1;   // queries per CTA
    const int i0 = PREFILL ? (int)blockIdx.y * qpc : 0;
    int p_begin, p_end;
    if (PREFILL) {
        p_begin = 0;
        p_end = max(0, min(kv_len, kv_len - seq_len + min(i0 + qpc, seq_len)));   // what the CTA's last query sees
    } else {
        int chunk_len = (kv_len + n_chunks - 1) / n_chunks;
        chunk_len = (chunk_len + 15) & ~15;
        p_begin = min(kv_len, chunk * chunk_len);
        p_end = min(kv_len, p_begin + chunk_len);
    }
    const size_t kv_dim = (size_t)num_kv_heads * HD;
    uint8_t *s_k = s_kv, *s_v = s_kv + FDM_SUPER * FDM_ROW;
    if (tid < FDM_SUPER / 16) mbar_init(&s_bar[tid], 32);   // 16 K-row + 16 V-row issuers per block
    mbar_fence_init();
    uint32_t phase = 0;
    const int my_row = tid & (FDM_SUPER - 1), my_is_v = tid >> 6;
    const int mi = lane >> 3, mr = lane & 7;   // ldmatrix: this lane addresses row mr of matrix mi

    for (int g0 = 0; g0 < group; g0 += 8) {
        const int heads_here = min(8, group - g0), head0 = kv_h * group + g0;
        const int cols = PREFILL ? heads_here * qpc : heads_here;   // live MMA columns: (query, head) pairs
        // column c -> (query c / heads_here, head c % heads_here); this thread's B-fragment column is g
        const int my_qi = g / heads_here, my_hh = g % heads_here;
        const bool col_live = g < cols && (!PREFILL || i0 + my_qi < seq_len);
        // query B fragments: column g, dims ks*16 + {2t, 2t+1} and + 8
        uint32_t qh[8][2], ql[8][2];
        float2 qv[8][2];
        const float *qrow = q + ((size_t)(PREFILL ? i0 + my_qi : 0) * num_heads + head0 + my_hh) * HD;
#pragma unroll
        for (int ks = 0; ks < 8; ks++)
#pragma unroll
            for (int hf = 0; hf < 2; hf++) {
                qv[ks][hf] = make_float2(0.f, 0.f);
                if (col_live) qv[ks][hf] = *reinterpret_cast<const float2 *>(qrow + ks * 16 + hf * 8 + 2 * t);
            }
        // the first rows are asked for before the queries have come (8 KV heads x 74 chunks at 4096 positions: with the factors of the
        // warps taken once below 7.7 -> 6.7 us in the step)
        auto ask = [&](int sp) {
            const int n_here = min(FDM_SUPER, p_end - sp);
            uint64_t *bar = &s_bar[my_row >> 4];
            if (my_row < n_here) {
                const uint16_t *src = (my_is_v ? v : k) + (size_t)(sp + my_row) * kv_dim + (size_t)kv_h * HD;
                mbar_arrive_expect_tx(bar, 2 * HD);
                bulk_g2s((my_is_v ? s_v : s_k) + my_row * FDM_ROW, src, 2 * HD, bar);
            } else {
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
            }
        };
        __syncthreads();   // everyone is done with the head pass before this one (and barrier init)
        if (p_begin < p_end) ask(p_begin);
#pragma unroll
        for (int ks = 0; ks < 8; ks++)
#pragma unroll
            for (int hf = 0; hf < 2; hf++) split_f16x2(qv[ks][hf].x * scale, qv[ks][hf].y * scale, qh[ks][hf], ql[ks][hf]);
        // causal limit of the two columns this thread owns in the score tile (2t, 2t+1)
        int lim[2] = {kv_len, kv_len};
        if (PREFILL) {
#pragma unroll
            for (int e = 0; e < 2; e++) lim[e] = kv_len - seq_len + i0 + (2 * t + e) / heads_here + 1;
        }
        float o[8][4];   // O^T tile mt: (dim 16mt+g | +8, head 2t | 2t+1)
#pragma unroll
        for (int n = 0; n < 8; n++) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
        float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};   // heads 2t, 2t+1 (l: this thread's share)

        for (int sp = p_begin; sp < p_end; sp += FDM_SUPER) {
            const int n_here = min(FDM_SUPER, p_end - sp);
            if (sp > p_begin) {
                __syncthreads();   // everyone is done with the previous pass's rows
                ask(sp);
            }
            const int rows = min(16, n_here - 16 * warp);
            if (rows > 0) {
                // rows past the end of a ragged block hold stale bytes: zero them so that a
                // masked probability (0) never meets a NaN/Inf pattern
                if (rows < 16) {
                    const int n_seg = (16 - rows) * 16;   // 16-byte segments per array
                    for (int i = lane; i < 2 * n_seg; i += 32) {
                        const int which = i / n_seg, j = i % n_seg;
                        uint8_t *row = (which ? s_v : s_k) + (16 * warp + rows + j / 16) * FDM_ROW;
                        *reinterpret_cast<uint4 *>(row + (j % 16) * 16) = make_uint4(0, 0, 0, 0);
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                }
                if (!mbar_wait_bounded(&s_bar[warp], phase)) {
                    if (lane == 0 && err_flag) atomicExch(err_flag, DEV_ERR_MBAR_TIMEOUT);
                } else {
                    // ---- S^T = K Q^T for this warp's 16 positions ----
                    float sc[4] = {0.f, 0.f, 0.f, 0.f};   // (pos g, head 2t) (g, 2t+1) (g+8, 2t) (g+8, 2t+1)
                    const uint32_t k_base = smem_u32(s_k) + (16 * warp + (mi & 1) * 8 + mr) * FDM_ROW + (mi >> 1) * 16;
#pragma unroll
                    for (int ks = 0; ks < 8; ks++) {
                        uint32_t a[4];
                        ldmatrix_x4(a, k_base + ks * 32);
                        mma_f16_16816(sc, a, qh[ks][0], qh[ks][1]);
                        mma_f16_16816(sc, a, ql[ks][0], ql[ks][1]);
                    }
                    if (g >= rows) sc[0] = sc[1] = -INFINITY;
                    if (g + 8 >= rows) sc[2] = sc[3] = -INFINITY;
                    if (PREFILL) {
                        const int pa = sp + 16 * warp + g;   // absolute position of rows g and g + 8
#pragma unroll
                        for (int e = 0; e < 2; e++) {
                            if (pa >= lim[e]) sc[e] = -INFINITY;
                            if (pa + 8 >= lim[e]) sc[2 + e] = -INFINITY;
                        }
                    }
                    // ---- online softmax per head (column): max over the 16 positions ----
                    float corr[2], pr[4];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        float mx = fmaxf(sc[e], sc[2 + e]);
                        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                        const float m_new = fmaxf(m_run[e], mx);   // stays -inf while everything is masked
                        corr[e] = m_run[e] == -INFINITY ? 0.f : expf(m_run[e] - m_new);
                        pr[e] = sc[e] == -INFINITY ? 0.f : expf(sc[e] - m_new);
                        pr[2 + e] = sc[2 + e] == -INFINITY ? 0.f : expf(sc[2 + e] - m_new);
                        l_run[e] = l_run[e] * corr[e] + (pr[e] + pr[2 + e]);
                        m_run[e] = m_new;
                    }
#pragma unroll
                    for (int n = 0; n < 8; n++) {
                        o[n][0] *= corr[0];
                        o[n][1] *= corr[1];
                        o[n][2] *= corr[0];
                        o[n][3] *= corr[1];
                    }
                    // P^T as B fragments: transpose the two 8x8 (pos x head) tiles across the warp
                    uint32_t p_lo_h, p_lo_l, p_hi_h, p_hi_l;
                    split_f16x2(pr[0], pr[1], p_lo_h, p_lo_l);   // positions 0..7
                    split_f16x2(pr[2], pr[3], p_hi_h, p_hi_l);   // positions 8..15
                    const uint32_t b0h = movmatrix_trans(p_lo_h), b0l = movmatrix_trans(p_lo_l);
                    const uint32_t b1h = movmatrix_trans(p_hi_h), b1l = movmatrix_trans(p_hi_l);
                    // ---- O^T += V^T P^T: A tiles are V[pos][dim] read transposed ----
                    const uint32_t v_base = smem_u32(s_v) + (16 * warp + (mi >> 1) * 8 + mr) * FDM_ROW + (mi & 1) * 16;
#pragma unroll
                    for (int mt = 0; mt < 8; mt++) {
                        uint32_t a[4];
                        ldmatrix_x4_trans(a, v_base + mt * 32);
                        mma_f16_16816(o[mt], a, b0h, b1h);
                        mma_f16_16816(o[mt], a, b0l, b1l);
                    }
                }
            }
            phase ^= 1;
        }
        // ---- merge the four warps (staging area reused as [warp][8 heads][128] f32) ----
#pragma unroll
        for (int e = 0; e < 2; e++) {
            l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 4);
            l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 8);
            l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], 16);
        }
        __syncthreads();
        float *s_acc = reinterpret_cast<float *>(s_kv);
#pragma unroll
        for (int mt = 0; mt < 8; mt++) {
            float *r0 = s_acc + (size_t)(warp * 8 + 2 * t) * FDM_ACC_STRIDE + mt * 16 + g;
            r0[0] = o[mt][0];
            r0[FDM_ACC_STRIDE] = o[mt][1];
            r0[8] = o[mt][2];
            r0[FDM_ACC_STRIDE + 8] = o[mt][3];
        }
        if (g == 0) {
#pragma unroll
            for (int e = 0; e < 2; e++) {
                s_ml[(warp * 8 + 2 * t + e) * 2] = m_run[e];
                s_ml[(warp * 8 + 2 * t + e) * 2 + 1] = l_run[e];
            }
        }
        __syncthreads();
        if (tid < 8 * (FDM_THREADS / 32)) {   // a warp's factor of a head: thread 8 warp + head
            const int hh = tid & 7;
            const float mw = s_ml[tid * 2];
            float M = -INFINITY;
#pragma unroll
            for (int w = 0; w < FDM_THREADS / 32; w++) M = fmaxf(M, s_ml[(w * 8 + hh) * 2]);
            s_factor[tid] = mw == -INFINITY ? 0.f : expf(mw - M);
            if (tid < 8) s_max[hh] = M;
        }
        __syncthreads();
        for (int hh = 0; hh < cols; hh++) {
            const int d = tid;
            const float M = s_max[hh];
            float a = 0.f, L = 0.f;
#pragma unroll
            for (int w = 0; w < FDM_THREADS / 32; w++) {
                const float f = s_factor[w * 8 + hh];
                a += s_acc[(size_t)(w * 8 + hh) * FDM_ACC_STRIDE + d] * f;
                L += s_ml[(w * 8 + hh) * 2 + 1] * f;
            }
            if (PREFILL) {
                const int qi = hh / heads_here;
                if (i0 + qi < seq_len) out[((size_t)(i0 + qi) * num_heads + head0 + hh % heads_here) * HD + d] = L > 0.f ? a / L : 0.f;
            } else {
                float *rec = partials + ((size_t)(head0 + hh) * n_chunks + chunk) * FD_PART_STRIDE;
                rec[d] = a;
                if (d == 0) {
                    rec[HD] = M;
                    rec[HD + 1] = L;
                }
            }
        }
        // the next head pass overwrites s_kv through the async proxy after these generic reads
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (!PREFILL && merge.cluster > 0) {
        // ---- all chunks of this KV head are one cluster: barrier, then CTA b merges the group's heads 2b, 2b + 1 ----
        __threadfence();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        const int hA = 2 * chunk;                       // first head of this CTA's pair within the group
        if (hA >= group) return;
        float *s_o = reinterpret_cast<float *>(s_kv);   // [2][128] merged rows
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 2; e++) {
            float o_val = 0.f;
            const int head = kv_h * group + hA + e;
            if (hA + e < group) {
                const float *base = partials + (size_t)head * n_chunks * FD_PART_STRIDE;
                float M = -INFINITY;
                for (int c = 0; c < n_chunks; c++) M = fmaxf(M, ld_l2(base + (size_t)c * FD_PART_STRIDE + HD));
                float a = 0.f, L = 0.f;
#pragma unroll 4
                for (int c = 0; c < n_chunks; c++) {
                    const float mc = ld_l2(base + (size_t)c * FD_PART_STRIDE + HD);
                    const float f = mc == -INFINITY ? 0.f : expf(mc - M);
                    L += ld_l2(base + (size_t)c * FD_PART_STRIDE + HD + 1) * f;
                    a += ld_l2(base + (size_t)c * FD_PART_STRIDE + tid) * f;
                }
                o_val = L > 0.f ? a / L : 0.f;
                if (merge.out) merge.out[(size_t)head * HD + tid] = o_val;
            }
            s_o[e * HD + tid] = o_val;
        }
        __syncthreads();
        if (merge.xq_out && warp == 0) {
            const float4 v0 = *(reinterpret_cast<const float4 *>(s_o) + 2 * lane), v1 = *(reinterpret_cast<const float4 *>(s_o) + 2 * lane + 1);
            const float vv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
            Q8kDevView dv = q8k_dev_view(merge.xq_out, num_heads * HD);
            const int blk = (kv_h * group) / 2 + chunk;
            q8k_quantize_block_warp(vv, lane, dv.qs + blk * 256, dv.d + blk, dv.bsum16 + blk * 16, nullptr);
        }
        return;
    }
    if (PREFILL || !merge.counters) return;
    // ---- last CTA of this KV head: merge its chunks --------------------------------------------
    __shared__ int s_last;
    __threadfence();   // this CTA's records are visible device-wide before it is counted
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&merge.counters[kv_h], 1) == n_chunks - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    float *s_f = reinterpret_cast<float *>(s_kv);                                   // [warp][n_chunks] rescale factors
    float *s_o = reinterpret_cast<float *>(s_kv) + (FDM_THREADS / 32) * FD_MAX_CHUNKS;   // [head of the group][128] merged rows
    static_assert(((FDM_THREADS / 32) * FD_MAX_CHUNKS + 16 * HD) * 4 <= FDM_KV_BYTES, "merge tail scratch must fit the staging area");
    float *my_f = s_f + warp * FD_MAX_CHUNKS;
    for (int g0 = 0; g0 < group; g0 += 16) {
        const int n_here = min(16, group - g0);
        // warp w merges heads w, w + 4, ... of this slice: lane = output dims 4 lane .. 4 lane + 3
        for (int hh = warp; hh < n_here; hh += FDM_THREADS / 32) {
            const int head = kv_h * group + g0 + hh;
            const float *base = partials + (size_t)head * n_chunks * FD_PART_STRIDE;
            float m = -INFINITY;
            for (int c = lane; c < n_chunks; c += 32) m = fmaxf(m, ld_l2(base + (size_t)c * FD_PART_STRIDE + HD));
            const float M = warp_max(m);
            float l = 0.f;
            for (int c = lane; c < n_chunks; c += 32) {
                const float mc = ld_l2(base + (size_t)c * FD_PART_STRIDE + HD);
                const float f = mc == -INFINITY ? 0.f : expf(mc - M);
                my_f[c] = f;
                l += ld_l2(base + (size_t)c * FD_PART_STRIDE + HD + 1) * f;
            }
            const float L = warp_sum(l);
            __syncwarp();
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int c = 0; c < n_chunks; c++) {
                // records are 130 floats apart: 8-byte alignment is all that holds for every chunk
                const float2 *rp = reinterpret_cast<const float2 *>(base + (size_t)c * FD_PART_STRIDE) + 2 * lane;
                const float2 r0 = ld_l2(rp), r1 = ld_l2(rp + 1);
                const float f = my_f[c];
                a.x += r0.x * f;
                a.y += r0.y * f;
                a.z += r1.x * f;
                a.w += r1.y * f;
            }
            const float4 o4 = L > 0.f ? make_float4(a.x / L, a.y / L, a.z / L, a.w / L) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (merge.out) *(reinterpret_cast<float4 *>(merge.out + (size_t)head * HD) + lane) = o4;
            *(reinterpret_cast<float4 *>(s_o + hh * HD) + lane) = o4;
            __syncwarp();
        }
        __syncthreads();
        if (merge.xq_out) {
            // heads 2b, 2b + 1 of the slice are one Q8_K block; the slice starts at an even head
            for (int bq = warp; 2 * bq + 1 < n_here; bq += FDM_THREADS / 32) {
                const float4 v0 = *(reinterpret_cast<const float4 *>(s_o + 2 * bq * HD) + 2 * lane), v1 = *(reinterpret_cast<const float4 *>(s_o + 2 * bq * HD) + 2 * lane + 1);
                const float vv[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
                Q8kDevView dv = q8k_dev_view(merge.xq_out, num_heads * HD);
                const int blk = (kv_h * group + g0) / 2 + bq;
                q8k_quantize_block_warp(vv, lane, dv.qs + blk * 256, dv.d + blk, dv.bsum16 + blk * 16, nullptr);
            }
        }
        __syncthreads();
    }
    if (tid == 0) merge.counters[kv_h] = 0;
}

RNB_GLOBAL void __launch_bounds__(FDM_THREADS, 4)
flash_decode_mma_kernel(const float *q, const uint16_t *k,
                        const uint16_t *v, const int *kv_len_dev,
                        int kv_len_host, int num_heads, int num_kv_heads, float scale,
                        float *partials, int *err_flag, const FdMerge merge) {
    fdm_body<false>(q, k, v, kv_len_dev, kv_len_host, 1, num_heads, num_kv_heads, scale, partials, nullptr, err_flag, merge);
}
// Causal prefill attention on the same machinery: grid (kv heads, ceil(seq / queries per CTA)).
RNB_GLOBAL void __launch_bounds__(FDM_THREADS, 4)
prefill_attention_mma_kernel(const float *q, const uint16_t *k, const uint16_t *v, int seq_len,
                             int kv_len, int num_heads, int num_kv_heads, float scale, float *out, int *err_flag) {
    fdm_body<true>(q, k, v, nullptr, kv_len, seq_len, num_heads, num_kv_heads, scale, nullptr, out, err_flag);
}

// Chunk merge: grid = num_heads, 512 threads.  The threads first agree on the global max and
// the per-chunk rescale factors (shared memory), then thread (group g = tid / 128, dim d) sums
// dimension d over the chunks c = g, g + 4, ...; the four groups are added at the end.  A head
// sharded onto one GPU of eight has hundreds of chunks: a serial walk would take tens of us.
RNB_GLOBAL void __launch_bounds__(4 * HD)
flash_decode_reduce_kernel(const float *partials, int n_chunks,
                           float *out, const PeerOut po = PeerOut{}) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float s_f[FD_MAX_CHUNKS];
    __shared__ float s_red[16];
    __shared__ float s_part[4][HD];
    const int h = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *base = partials + (size_t)h * n_chunks * FD_PART_STRIDE;
    float m = -INFINITY;
    for (int c = tid; c < n_chunks; c += 4 * HD) m = fmaxf(m, base[(size_t)c * FD_PART_STRIDE + HD]);
    m = warp_max(m);
    if (lane == 0) s_red[warp] = m;
    __syncthreads();
    float M = -INFINITY;
#pragma unroll
    for (int i = 0; i < 16; i++) M = fmaxf(M, s_red[i]);
    __syncthreads();
    float l = 0.f;
    for (int c = tid; c < n_chunks; c += 4 * HD) {
        const float mc = base[(size_t)c * FD_PART_STRIDE + HD];
        const float f = mc == -INFINITY ? 0.f : expf(mc - M);
        s_f[c] = f;
        l += base[(size_t)c * FD_PART_STRIDE + HD + 1] * f;
    }
    l = warp_sum(l);
    if (lane == 0) s_red[warp] = l;
    __syncthreads();
    float L = 0.f;
#pragma unroll
    for (int i = 0; i < 16; i++) L += s_red[i];
    const int g = tid >> 7, d = tid & (HD - 1);
    float a = 0.f;
#pragma unroll 8
    for (int c = g; c < n_chunks; c += 4) a += base[(size_t)c * FD_PART_STRIDE + d] * s_f[c];
    s_part[g][d] = a;
    __syncthreads();
    if (g == 0) {
        const float t = (s_part[0][d] + s_part[1][d]) + (s_part[2][d] + s_part[3][d]);
        const float o = L > 0.f ? t / L : 0.f;
        out[(size_t)h * HD + d] = o;
        if (po.peers) {
            // sharded decode: the head's row also goes straight into every peer's gathered buffer
            peer_store(po, (size_t)h * HD + d, o);
            __threadfence_system();
        }
    }
    if (po.peers) {
        __syncthreads();
        if (tid == 0) peer_arrive(po);
    }
}

// Chunk merge fused with the Q8_K quantisation of the attention output (the o_proj input); two heads are exactly one 256-element
// block.  A cluster of eight CTAs per block: CTA r merges 32 output dims of head r / 4 of the two.  A warp sums every eighth
// chunk's records, a lane a dim, the eight sums are added in a fixed order; CTA 0 quantises.  The records of the first FDR_AHEAD
// chunks of each warp are asked for together with the maxima and sums: one round trip to L2.
// What bounds it: that round trip, the launch and two cluster barriers.  32 heads x 74 chunks in the step: 4.3 us; one CTA of 1024
// threads per block, the maxima first: 7.1.
constexpr int FDR_CTAS = 8, FDR_THREADS = 256, FDR_AHEAD = 10;
RNB_GLOBAL void __launch_bounds__(FDR_THREADS)
flash_decode_reduce_q8k_cluster_kernel(const float *partials, int n_chunks, int num_heads, uint8_t *xq_out) {
    pdl_launch_dependents();
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    pdl_wait();
    __shared__ __align__(16) float s_out[2 * HD];
    __shared__ float s_f[FD_MAX_CHUNKS];
    __shared__ float s_red[2][FDR_THREADS / 32];
    __shared__ float s_part[FDR_THREADS / 32][32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)blockIdx.x % FDR_CTAS, block = (int)blockIdx.x / FDR_CTAS;
    const int hs = rank >> 2, d = (rank & 3) * 32 + lane;
    const float *base = partials + (size_t)(2 * block + hs) * n_chunks * FD_PART_STRIDE;
    float ahead[FDR_AHEAD];
#pragma unroll
    for (int i = 0; i < FDR_AHEAD; i++) {
        const int c = warp + 8 * i;
        ahead[i] = c < n_chunks ? base[(size_t)c * FD_PART_STRIDE + d] : 0.f;
    }
    float m = -INFINITY;
    const float2 own = tid < n_chunks ? *reinterpret_cast<const float2 *>(base + (size_t)tid * FD_PART_STRIDE + HD) : make_float2(-INFINITY, 0.f);
    m = own.x;
    for (int c = tid + FDR_THREADS; c < n_chunks; c += FDR_THREADS) m = fmaxf(m, base[(size_t)c * FD_PART_STRIDE + HD]);
    m = warp_max(m);
    if (lane == 0) s_red[0][warp] = m;
    __syncthreads();
    float M = s_red[0][0];
#pragma unroll
    for (int i = 1; i < FDR_THREADS / 32; i++) M = fmaxf(M, s_red[0][i]);
    float l = 0.f;
    for (int c = tid; c < n_chunks; c += FDR_THREADS) {
        const float2 ml = c == tid ? own : *reinterpret_cast<const float2 *>(base + (size_t)c * FD_PART_STRIDE + HD);
        const float f = ml.x == -INFINITY ? 0.f : expf(ml.x - M);
        s_f[c] = f;
        l += ml.y * f;
    }
    l = warp_sum(l);
    if (lane == 0) s_red[1][warp] = l;
    __syncthreads();
    float a = 0.f;
#pragma unroll
    for (int i = 0; i < FDR_AHEAD; i++) {
        const int c = warp + 8 * i;
        if (c < n_chunks) a += ahead[i] * s_f[c];
    }
#pragma unroll 8
    for (int c = warp + 8 * FDR_AHEAD; c < n_chunks; c += 8) a += base[(size_t)c * FD_PART_STRIDE + d] * s_f[c];
    s_part[warp][lane] = a;
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // every CTA of the cluster runs: CTA 0's memory may be written
    if (warp == 0) {
        float t = 0.f, L = 0.f;
#pragma unroll
        for (int i = 0; i < FDR_THREADS / 32; i++) t += s_part[i][lane], L += s_red[1][i];
        ps_st_remote(ps_map(smem_u32(s_out + hs * HD + d), 0), __float_as_uint(L > 0.f ? t / L : 0.f));
    }
    __syncwarp();
    ps_cluster_sync();
    if (rank == 0 && warp == 0) {
        const float4 v0 = *reinterpret_cast<const float4 *>(s_out + lane * 8), v1 = *reinterpret_cast<const float4 *>(s_out + lane * 8 + 4);
        const float v[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        Q8kDevView dv = q8k_dev_view(xq_out, num_heads * HD);
        q8k_quantize_block_warp(v, lane, dv.qs + block * 256, dv.d + block, dv.bsum16 + block * 16, nullptr);
    }
}

// ---------------------------------------------------------------------------------------------
// Reference-order decode attention: the same floating-point operations in the same order as
// rnb-cpu's four-pass decode kernel (crates/rnb-cpu/src/kernels/attention/decode_flash.rs:91-212
// with the f32·f16 helpers of x86_helpers.rs:11-80), so the result is bit-identical to the CPU's:
//   score_j = hsum(16 lanes, each 8 sequential mul-then-add steps over dims 16i + lane) * scale
//   m = max_j score_j;  p_j = expf(score_j - m);  sum = ((p_0 + p_1) + p_2) + ...  (f32, in order)
//   w_j = p_j * (1 / sum);  out_d = ((v_0d * w_0) + v_1d * w_1) + ...              (mul, then add)
// The chunked tensor-core kernel above reassociates all three sums; its result differs in the last
// bits, which the Q8_K rounding of the o_proj input can amplify.  This kernel is the one used for
// short contexts, where the in-order sums cost less than a microsecond.
//
// expf is the C library's on the reference's platform: glibc's single-precision routine evaluates
// 2^(k/32) * P(r) in binary64 (a 32-entry table of 2^(i/32) and a cubic in r) and rounds once to
// f32.  The same evaluation here agrees with it on every input up to the binary64 rounding of
// intermediate steps, which is 2^29 times finer than an f32 ulp.
//
// Two heads (a Q8_K block of the output) belong to a cluster of eight CTAs.  A CTA computes the scores of an eighth of the
// positions for both heads and hands them to the four CTAs of each head; a CTA then takes the softmax of its head, which needs all
// scores, and 32 of the head's output dims: products by all threads, sums over the positions by one warp.  Values travel into
// shared memory while the softmax runs.
//
// What bounds it: a chain of latencies (launch, one round trip for keys, three cluster barriers, 1000 cycles each) and the two sums
// in position order, four to six cycles a position each.  In the step of 16 heads on 8 KV heads: 6.5 us at 100 positions, 11.5 at 345
// (two heads per CTA, without a cluster: 7.4 and 22.3).
// ---------------------------------------------------------------------------------------------
constexpr int AX_CTAS = 8, AX_THREADS = 256;
constexpr int AX_MAX_LEN = 4096;      // scores of a head: 16 KB
constexpr int AX_SLAB = 512;          // positions of V at a time, 32 dims each
// pitches: of a position's values (80 bytes), of a dim's products (516): four threads, eight threads apart in the banks
constexpr int AX_ROW = 80, AX_COL = AX_SLAB + 4;
constexpr uint32_t AX_PROD = AX_SLAB * AX_ROW, AX_SCORES = AX_PROD + 32 * AX_COL * 4;
inline size_t ax_smem_bytes(int max_len) { return (size_t)AX_SCORES + (size_t)(max_len + 16) * sizeof(float); }   // reads run ahead by a group of 16

__device__ __forceinline__ void ax_copy16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// positions pos0.. of 32 dims (64 bytes a position) into the slab
__device__ __forceinline__ void ax_fetch_values(uint8_t *slab, const uint16_t *v, size_t kv_dim, int pos0, int n, int tid) {
    for (int i = tid; i < 4 * n; i += AX_THREADS) ax_copy16(slab + AX_ROW * (i >> 2) + 16 * (i & 3), v + (size_t)(pos0 + (i >> 2)) * kv_dim + 8 * (i & 3));
}
// start + x[0] + x[1] + ... in order; the next sixteen on their way while these are added
__device__ __forceinline__ float ax_sum(const float *x, int n, float start) {
    float4 next[4];
#pragma unroll
    for (int u = 0; u < 4; u++) next[u] = *reinterpret_cast<const float4 *>(x + 4 * u);   // past the end: not used
    int j = 0;
    for (; j + 16 <= n; j += 16) {
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; u++) p[u] = next[u];
        if (j + 32 <= n) {
#pragma unroll
            for (int u = 0; u < 4; u++) next[u] = *reinterpret_cast<const float4 *>(x + j + 16 + 4 * u);
        }
#pragma unroll
        for (int u = 0; u < 4; u++) start = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(start, p[u].x), p[u].y), p[u].z), p[u].w);
    }
    for (; j < n; j++) start = __fadd_rn(start, x[j]);
    return start;
}
__device__ __forceinline__ void ax_values_landed() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// grid = AX_CTAS x ceil(num_heads / 2), cluster (AX_CTAS, 1, 1); dynamic shared memory = ax_smem_bytes(max_len).  Writes `out`
// ([num_heads][128] f32) and/or the Q8_K blocks of the output (`xq_out`, needs an even head
// count: two heads are one 256-element block).  K and V must be 16-byte aligned.  A context
// longer than max_len raises the error flag and writes nothing.
RNB_GLOBAL void __launch_bounds__(AX_THREADS)
attention_decode_exact_kernel(const float *q, const uint16_t *k, const uint16_t *v, const int *kv_len_dev, int kv_len_host, int max_len, int num_heads,
                              int num_kv_heads, float scale, float *out, uint8_t *xq_out, int *err_flag) {
    pdl_launch_dependents();
    extern __shared__ __align__(16) uint8_t s_dyn[];
    uint8_t *const slab = s_dyn;                                              // [position][32 dims]
    float *const prod = reinterpret_cast<float *>(s_dyn + AX_PROD);           // [32 dims][position]
    float *const sc = reinterpret_cast<float *>(s_dyn + AX_SCORES);           // [max_len]
    __shared__ unsigned long long s_tab[32];
    __shared__ float s_red[AX_THREADS / 32];
    __shared__ float s_inv;
    __shared__ __align__(16) float s_o[2 * HD];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)blockIdx.x % AX_CTAS;
    if (tid < 32) s_tab[tid] = c_exp2_tab32[tid];
    const int group = num_heads / num_kv_heads;
    const size_t kv_dim = (size_t)num_kv_heads * HD;
    const int h0 = ((int)blockIdx.x / AX_CTAS) * 2, h1 = min(h0 + 1, num_heads - 1);   // an odd head count repeats the last head
    const size_t off0 = (size_t)(h0 / group) * HD, off1 = (size_t)(h1 / group) * HD;
    const bool shared_kv = off0 == off1;
    const int hs = rank >> 2, d0 = (rank & 3) * 32;                           // this CTA's head, its output dims
    asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");
    pdl_wait();
    const int kv_len = kv_len_dev ? *kv_len_dev + kv_len_host : kv_len_host;
    if (kv_len < 1 || kv_len > max_len) {
        if (tid == 0 && err_flag) atomicExch(err_flag, DEV_ERR_BAD_JOB);
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        return;
    }
    const uint16_t *const vh = v + (hs ? off1 : off0) + d0;
    ax_fetch_values(slab, vh, kv_dim, 0, min(kv_len, AX_SLAB), tid);

    // pass 1: scores.  Half-warp (16 lanes) per position, lane l owns dims 16 i + l; four positions' rows in flight.
    {
        const int l16 = lane & 15, hw = tid >> 4, per = (kv_len + AX_CTAS - 1) / AX_CTAS, first = rank * per, last = min(kv_len, first + per);
        float qa[8], qb[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            qa[i] = q[(size_t)h0 * HD + 16 * i + l16];
            qb[i] = q[(size_t)h1 * HD + 16 * i + l16];
        }
        // lanes 0-3 hand the first head's score to CTAs 0-3, lanes 4-7 the second's to CTAs 4-7
        const uint32_t to = ps_map(smem_u32(sc), l16 & 7);
        bool others = false;
        auto wait_for_others = [&]() {   // every CTA of the cluster runs: its memory may be written
            if (!others) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
            others = true;
        };
        for (int b = first; b < last; b += 4 * (AX_THREADS / 16)) {   // the same trips for all threads
            const int j0 = b + hw;
            uint16_t ka[4][8], kb[4][8];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int j = min(j0 + u * (AX_THREADS / 16), last - 1);
                const uint16_t *row = k + (size_t)j * kv_dim + l16;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    ka[u][i] = row[off0 + 16 * i];
                    kb[u][i] = shared_kv ? ka[u][i] : row[off1 + 16 * i];
                }
            }
            wait_for_others();
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int j = j0 + u * (AX_THREADS / 16);
                if (b + u * (AX_THREADS / 16) >= last) break;
                float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    acc0 = __fadd_rn(acc0, __fmul_rn(qa[i], __half2float(__ushort_as_half(ka[u][i]))));
                    acc1 = __fadd_rn(acc1, __fmul_rn(qb[i], __half2float(__ushort_as_half(kb[u][i]))));
                }
                // lanes l and l + 8 are the reference's two accumulators; then lo + hi, movehdup, movehl
#pragma unroll
                for (int o = 8; o >= 4; o >>= 1) {
                    acc0 = __fadd_rn(acc0, __shfl_xor_sync(0xffffffffu, acc0, o));
                    acc1 = __fadd_rn(acc1, __shfl_xor_sync(0xffffffffu, acc1, o));
                }
                acc0 = __fadd_rn(acc0, __shfl_xor_sync(0xffffffffu, acc0, 1));
                acc1 = __fadd_rn(acc1, __shfl_xor_sync(0xffffffffu, acc1, 1));
                acc0 = __fadd_rn(acc0, __shfl_xor_sync(0xffffffffu, acc0, 2));
                acc1 = __fadd_rn(acc1, __shfl_xor_sync(0xffffffffu, acc1, 2));
                if (l16 < AX_CTAS && j < last) ps_st_remote(to + 4u * (uint32_t)j, __float_as_uint(__fmul_rn(l16 < 4 ? acc0 : acc1, scale)));
            }
        }
        wait_for_others();
    }
    __syncwarp();
    ps_cluster_sync();
    // pass 2: max
    float m = -INFINITY;
    for (int j = tid; j < kv_len; j += AX_THREADS) m = fmaxf(m, sc[j]);
    m = warp_max(m);
    if (lane == 0) s_red[warp] = m;
    __syncthreads();
    float M = s_red[0];
#pragma unroll
    for (int i = 1; i < AX_THREADS / 32; i++) M = fmaxf(M, s_red[i]);
    // pass 3: exponentials in parallel, their sum in position order by one thread
    for (int j = tid; j < kv_len; j += AX_THREADS) sc[j] = expf_libm_smem(__fsub_rn(sc[j], M), s_tab);
    __syncthreads();
    if (tid == 0) {
        const float sum = ax_sum(sc, kv_len, 0.0f);
        s_inv = sum > 0.0f ? __fdiv_rn(1.0f, sum) : 0.0f;
    }
    __syncthreads();
    // pass 4: weights times values in parallel, their sum in position order by one thread per output dim
    const float inv = s_inv;
    float o = 0.0f;
    for (int pos0 = 0; pos0 < kv_len; pos0 += AX_SLAB) {
        const int n = min(AX_SLAB, kv_len - pos0);
        if (pos0 > 0) ax_fetch_values(slab, vh, kv_dim, pos0, n, tid);
        ax_values_landed();
        __syncthreads();                                                      // values landed; the products before these have been read
        for (int p = lane; p < n; p += 32) {                                  // four dims of a position
            const uint2 x = *reinterpret_cast<const uint2 *>(slab + AX_ROW * p + 8 * warp);
            const float w = __fmul_rn(sc[pos0 + p], inv);
            const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&x.x)), c = __half22float2(*reinterpret_cast<const __half2 *>(&x.y));
            float *to = prod + 4 * warp * AX_COL + p;
            to[0] = __fmul_rn(a.x, w), to[AX_COL] = __fmul_rn(a.y, w), to[2 * AX_COL] = __fmul_rn(c.x, w), to[3 * AX_COL] = __fmul_rn(c.y, w);
        }
        __syncthreads();
        if (warp == 0) o = ax_sum(prod + lane * AX_COL, n, o);
    }
    const int h = h0 + hs;
    const bool live = h < num_heads;
    if (warp == 0) {
        if (live && out) out[(size_t)h * HD + d0 + lane] = o;
        if (xq_out) ps_st_remote(ps_map(smem_u32(s_o + hs * HD + d0 + lane), 0), __float_as_uint(live ? o : 0.0f));
    }
    if (!xq_out) return;
    ps_cluster_sync();
    if (rank == 0 && tid < 32) {
        const float4 v0 = *reinterpret_cast<const float4 *>(s_o + lane * 8), v1 = *reinterpret_cast<const float4 *>(s_o + lane * 8 + 4);
        const float vals[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        Q8kDevView dv = q8k_dev_view(xq_out, num_heads * HD);
        const int b = (int)blockIdx.x / AX_CTAS;
        q8k_quantize_block_warp(vals, lane, dv.qs + b * 256, dv.d + b, dv.bsum16 + b * 16, nullptr);
    }
}

}  // namespace rnb
