// Causal prefill attention on the 5th-generation tensor cores: one CTA owns 128 (query, head) rows of one KV head -
// 128 / group consecutive query positions x the group's heads - and walks the visible keys in tiles of 64.  Arithmetic:
// f16 operands, fp32 accumulators; q and the probabilities enter as f16 "hi" + f16 remainder "lo" so that the products
// keep fp32-level accuracy against the f16 cache; softmax(q.K^T * scale).V per head with the online maximum, as
// rnb-cpu's attention_with_scale_window_and_softcap (crates/rnb-cpu/src/kernels/attention/batch_f32.rs:76+); query i sees
// keys 0 .. kv_len - seq_len + i.
//
// Row r = (query r / group, head r % group) is tensor-memory lane r and belongs to one thread of warps 0-3: a row's maximum
// and sum need no shuffles.  Warp 4 issues the products: scores (128 rows x 64 keys, queries and keys from shared memory), then
// probabilities from tensor memory x values.  The scores of tile t + 1 are under way while the softmax of tile t runs.  Warp 5
// copies K and V tiles into a ring of three 16 KB slots in the order of their use (K0 K1 V0 K2 V1 ...).  The output stays in
// tensor memory; it is scaled only when a row's maximum has grown by more than a factor 2^8 over the one in use, so that
// probabilities are at most 2^8.  Two CTAs per SM (112 KB, 256 tensor-memory columns each: 64 scores, 128 outputs, 32 + 32
// probabilities).  Long rows are scheduled first.  Every wait is bounded.
//
// What bounds it: the softmax warps.  Caches warm, 32 / 8 heads: 2048 tokens 76 us (247 with mma.sync and eight warps that shared a
// CTA), 203 tokens behind 1000 positions 31 (65); 64 tokens of 8 / 2 heads 10.3 (7.9: the fill of tensor memory and barriers).
#pragma once
#include "attention.cuh"
#include "prefill_gemm_split.cuh"

namespace rnb {

constexpr int PAT_ROWS = 128;                      // (query, head) rows per CTA
constexpr int PAT_KEYS = 64;                       // keys per tile
constexpr int PAT_THREADS = 192;
constexpr int PAT_SLOTS = 3;
constexpr uint32_t PAT_PANEL = PAT_ROWS * 128;     // 64 dims of the queries, 128-byte swizzle
constexpr uint32_t PAT_Q_BYTES = 4 * PAT_PANEL;    // hi, lo x two panels
constexpr uint32_t PAT_TILE_BYTES = PAT_KEYS * 2 * HD;
constexpr size_t PAT_SMEM = PAT_Q_BYTES + PAT_SLOTS * PAT_TILE_BYTES + 128;   // + barriers; two CTAs per SM leave no room to align
constexpr float PAT_GROWTH = 8.0f;                 // log2

struct PatMaps {
    PgTensorMap k, v;   // [kv_len][kv heads * 128] f16, boxes of 64 columns x 64 rows
};

// V as the second operand: dims contiguous ("MN-major"), 128-byte swizzle: 8 keys x 64 dims are 1024 bytes, the next 8 keys follow,
// the other 64 dims are a panel of 64 keys further
__device__ __forceinline__ uint64_t pat_v_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)((PAT_KEYS * 128) >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// D = f32, A = B = f16, M = 128
constexpr uint32_t PAT_IDESC_S = (1u << 4) | ((uint32_t)(PAT_KEYS >> 3) << 17) | ((uint32_t)(PAT_ROWS >> 4) << 24);
constexpr uint32_t PAT_IDESC_O = (1u << 4) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(PAT_ROWS >> 4) << 24);   // second operand MN-major
// D += A (tensor memory) x B
__device__ __forceinline__ void pat_mma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void pat_tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
        "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void pat_tmem_ld64(uint32_t taddr, uint32_t (&v)[64]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,"
        "%61,%62,%63}, [%64];\n\ttcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
          "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),
          "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31]), "=r"(v[32]), "=r"(v[33]),
          "=r"(v[34]), "=r"(v[35]), "=r"(v[36]), "=r"(v[37]), "=r"(v[38]), "=r"(v[39]), "=r"(v[40]), "=r"(v[41]), "=r"(v[42]), "=r"(v[43]), "=r"(v[44]),
          "=r"(v[45]), "=r"(v[46]), "=r"(v[47]), "=r"(v[48]), "=r"(v[49]), "=r"(v[50]), "=r"(v[51]), "=r"(v[52]), "=r"(v[53]), "=r"(v[54]), "=r"(v[55]),
          "=r"(v[56]), "=r"(v[57]), "=r"(v[58]), "=r"(v[59]), "=r"(v[60]), "=r"(v[61]), "=r"(v[62]), "=r"(v[63])
        : "r"(taddr)
        : "memory");
}
// 2^x; what is below 2^-126 of the largest probability is zero
__device__ __forceinline__ float pat_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// packed f32: {x, y} * m + a, and sums; each half rounds as the single operation does
__device__ __forceinline__ float2 pat_fma2(float x, float y, uint64_t m, uint64_t a) {
    float2 r;
    asm("{\n\t.reg .b64 t;\n\tmov.b64 t, {%2, %3};\n\tfma.rn.f32x2 t, t, %4, %5;\n\tmov.b64 {%0, %1}, t;\n\t}" : "=f"(r.x), "=f"(r.y) : "f"(x), "f"(y), "l"(m), "l"(a));
    return r;
}
__device__ __forceinline__ void pat_add2(uint64_t &sum, float x, float y) {
    asm("{\n\t.reg .b64 t;\n\tmov.b64 t, {%1, %2};\n\tadd.rn.f32x2 %0, %0, t;\n\t}" : "+l"(sum) : "f"(x), "f"(y));
}
__device__ __forceinline__ float pat_total(uint64_t a, uint64_t b) {
    return (__uint_as_float((uint32_t)a) + __uint_as_float((uint32_t)(a >> 32))) + (__uint_as_float((uint32_t)b) + __uint_as_float((uint32_t)(b >> 32)));
}
__device__ __forceinline__ void pat_tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// grid = num_kv_heads x ceil(seq_len / (128 / group)), heads fastest: the long rows of every head come first; group =
// num_heads / num_kv_heads a power of two up to 128.  The softmax needs a positive scale (its maxima are of unscaled scores): the
// sign, or zero, of another one goes into the queries.  out_bf16 (may be null): the result rounded to bf16 there instead of f32 in `out`.
RNB_GLOBAL void __launch_bounds__(PAT_THREADS, 2)
prefill_attention_tiled_kernel(const float *q, const __grid_constant__ PatMaps maps, int seq_len, int kv_len, int num_heads, int num_kv_heads,
                               float scale, float *out, uint16_t *out_bf16, int *err_flag) {
    extern __shared__ __align__(1024) uint8_t pat_smem[];
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint64_t *const bars = reinterpret_cast<uint64_t *>(pat_smem + PAT_Q_BYTES + PAT_SLOTS * PAT_TILE_BYTES);
    uint64_t *const full = bars, *const empty = bars + PAT_SLOTS, *const q_full = bars + 6, *const s_full = bars + 7, *const s_free = bars + 8, *const p_full = bars + 9,
                    *const pv_done = bars + 10;
    volatile uint32_t *const tmem_slot = reinterpret_cast<volatile uint32_t *>(bars + 11);
    volatile int *const s_failed = reinterpret_cast<volatile int *>(bars + 12);
    const uint32_t smem = smem_u32(pat_smem);
    const int group = num_heads / num_kv_heads, qpc = PAT_ROWS / group;
    const int kv_h = (int)blockIdx.x % num_kv_heads, i0 = (((int)gridDim.x - 1 - (int)blockIdx.x) / num_kv_heads) * qpc;   // long rows first
    const int shift = kv_len - seq_len;                                              // query i sits at position shift + i
    const int n_keys = min(kv_len, shift + min(i0 + qpc, seq_len));                  // keys visible to the CTA's last query
    const int n_tiles = (n_keys + PAT_KEYS - 1) / PAT_KEYS;
    if (tid == 0) {
        for (int s = 0; s < PAT_SLOTS; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(q_full, 4);
        mbar_init(s_full, 1);
        mbar_init(s_free, 4);
        mbar_init(p_full, 4);
        mbar_init(pv_done, 1);
        mbar_fence_init();
        *s_failed = (smem & 1023u) != 0;
    }
    pdl_wait();   // the queries and the cache are the previous launch's result; tensor memory is asked for when no earlier launch can still hold it
    if (warp == 4) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t *>(tmem_slot))), "r"(256) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    pg_fence_before();
    __syncthreads();
    pg_fence_after();
    const uint32_t tmem = *tmem_slot, t_s = tmem, t_o = tmem + 64, t_ph = tmem + 192, t_pl = tmem + 224;
    bool ok = *s_failed == 0;

    if (warp < 4) {
        // ---- queries as f16 hi + lo: a warp takes its 32 rows, four dims per lane, 16 rows asked for at once (one by one the rows took
        // 13 us, most of a short prompt's launch) ----
        const float sign = scale > 0.f ? 1.f : scale == 0.f ? 0.f : -1.f;
        for (int i = 0; i < 32 && ok; i += 16) {
            float4 x[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int r = warp * 32 + i + j, qi = i0 + r / group;
                x[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (qi < seq_len) x[j] = *reinterpret_cast<const float4 *>(q + ((size_t)qi * num_heads + kv_h * group + r % group) * HD + lane * 4);
            }
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int r = warp * 32 + i + j;
                uint2 hi, lo;
                split_f16x2(x[j].x * sign, x[j].y * sign, hi.x, lo.x);
                split_f16x2(x[j].z * sign, x[j].w * sign, hi.y, lo.y);
                const uint32_t at = (uint32_t)(lane >> 4) * PAT_PANEL + (uint32_t)(r >> 3) * 1024u + (uint32_t)(r & 7) * 128u +
                                    (((uint32_t)((lane & 15) >> 1) ^ (uint32_t)(r & 7)) << 4) + (uint32_t)(lane & 1) * 8u;
                *reinterpret_cast<uint2 *>(pat_smem + at) = hi;
                *reinterpret_cast<uint2 *>(pat_smem + 2 * PAT_PANEL + at) = lo;
            }
        }
        pg_proxy_fence();
        __syncwarp();
        if (lane == 0) pg_arrive(q_full);
        // ---- softmax: this thread's row ----
        const int r = warp * 32 + lane, qi = i0 + r / group;
        const bool live = qi < seq_len;
        const int pos = live ? shift + qi : kv_len - 1;   // dead rows see everything (finite numbers) and are never stored
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        const float sl2 = scale == 0.f ? 1.f : fabsf(scale) * 1.4426950408889634f;   // scores are kept in log2 units: exp(x) = exp2(x * log2 e)
        float m_ref = -INFINITY, l_run = 0.f;
        for (int t = 0; t < n_tiles && ok; t++) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(s_full, (uint32_t)(t & 1)));
            if (!ok) break;
            pg_fence_after();
            uint32_t s[PAT_KEYS];
            pat_tmem_ld64(t_s + lanes, s);
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pg_arrive(s_free);
            const int seen = pos - t * PAT_KEYS;   // the tile's keys 0 .. seen are visible
            if (seen < PAT_KEYS - 1) {
#pragma unroll
                for (int i = 0; i < PAT_KEYS; i++)
                    if (i > seen) s[i] = 0xff800000u;   // -inf
            }
            float mxs[4];
#pragma unroll
            for (int j = 0; j < 4; j++) mxs[j] = __uint_as_float(s[j]);
#pragma unroll
            for (int i = 4; i < PAT_KEYS; i++) mxs[i & 3] = fmaxf(mxs[i & 3], __uint_as_float(s[i]));
            const float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])) * sl2;   // sl2 > 0
            // the maximum in use; the output is scaled when it falls behind by more than PAT_GROWTH
            float corr = 1.0f;
            if (mx > m_ref + PAT_GROWTH || m_ref == -INFINITY) {
                const float m_new = fmaxf(mx, m_ref);
                corr = exp2f(m_ref - (m_new == -INFINITY ? 0.f : m_new));   // exp2(-inf) = 0 on the first tile
                m_ref = m_new;
            }
            const float m_use = m_ref == -INFINITY ? 0.f : m_ref;   // a fully masked row so far: keep everything at zero
            const uint64_t sl22 = pg_pair_f32(sl2, sl2), nm2 = pg_pair_f32(-m_use, -m_use);
            uint64_t sum[2] = {0, 0};
            uint32_t ph[32], pl[32];
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const float2 x = pat_fma2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]), sl22, nm2);
                const float p0 = pat_exp2(x.x), p1 = pat_exp2(x.y);
                pat_add2(sum[i & 1], p0, p1);
                split_f16x2(p0, p1, ph[i], pl[i]);
            }
            l_run = fmaf(l_run, corr, pat_total(sum[0], sum[1]));
            if (t > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(pv_done, (uint32_t)((t - 1) & 1)));   // the probabilities' columns are free, the output stands
                if (!ok) break;
                pg_fence_after();
                if (__any_sync(0xffffffffu, corr != 1.0f)) {
#pragma unroll 1
                    for (int c = 0; c < 4; c++) {
                        uint32_t v[32];
                        pg_tmem_ld32(t_o + lanes + (uint32_t)c * 32u, v);
#pragma unroll
                        for (int i = 0; i < 32; i++) v[i] = __float_as_uint(__uint_as_float(v[i]) * corr);
                        pat_tmem_st32(t_o + lanes + (uint32_t)c * 32u, v);
                    }
                }
            }
            __syncwarp();
            pat_tmem_st32(t_ph + lanes, ph);
            pat_tmem_st32(t_pl + lanes, pl);
            pat_tmem_st_wait();
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pg_arrive(p_full);
        }
        if (ok && n_tiles > 0) ok = __all_sync(0xffffffffu, mbar_wait_bounded(pv_done, (uint32_t)((n_tiles - 1) & 1)));
        if (ok) {
            pg_fence_after();
            const float inv = l_run > 0.f ? 1.0f / l_run : 0.f;
            const size_t at = ((size_t)min(qi, seq_len - 1) * num_heads + kv_h * group + r % group) * HD;
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                uint32_t v[32];
                pg_tmem_ld32(t_o + lanes + (uint32_t)c * 32u, v);
                if (!live) continue;
                auto o = [&](int i) { return __uint_as_float(v[i]) * inv; };
                if (out_bf16) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8)
                        *reinterpret_cast<uint4 *>(out_bf16 + at + c * 32 + i) =
                            make_uint4(pg_pack_bf16(o(i), o(i + 1)), pg_pack_bf16(o(i + 2), o(i + 3)), pg_pack_bf16(o(i + 4), o(i + 5)), pg_pack_bf16(o(i + 6), o(i + 7)));
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4 *>(out + at + c * 32 + i) = make_float4(o(i), o(i + 1), o(i + 2), o(i + 3));
                }
            }
        }
    } else if (warp == 4) {
        // ---- products; item i of the ring lies in slot i % 3 ----
        const uint32_t ring = smem + PAT_Q_BYTES;
        uint32_t it = 0;
        auto arrived = [&]() { return __all_sync(0xffffffffu, mbar_wait_bounded(&full[it % PAT_SLOTS], (it / PAT_SLOTS) & 1u)); };
        auto scores = [&]() {   // of the K tile that is next in the ring
            ok = ok && arrived();
            if (!ok) return;
            pg_fence_after();
            if (pg_elect()) {
                const uint32_t kt = ring + (it % PAT_SLOTS) * PAT_TILE_BYTES;
#pragma unroll
                for (int part = 1; part >= 0; part--)   // lo before hi: the accumulator truncates what it adds, and adds less often to full sums
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const uint64_t dq = pg_smem_desc(smem + (uint32_t)(2 * part + p) * PAT_PANEL), dk = pg_smem_desc(kt + (uint32_t)p * (PAT_KEYS * 128));
#pragma unroll
                        for (int k = 0; k < 4; k++) ps_mma(t_s, dq + 2u * k, dk + 2u * k, PAT_IDESC_S, (1 - part) | p | k);   // 16 dims, 32 bytes on
                    }
                pg_commit(&empty[it % PAT_SLOTS]);
                pg_commit(s_full);
            }
            __syncwarp();
            it++;
        };
        if (n_tiles > 0) {
            ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(q_full, 0u));
            scores();
        }
        for (int t = 0; t < n_tiles && ok; t++) {
            if (t + 1 < n_tiles) {
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(s_free, (uint32_t)(t & 1)));
                scores();
            }
            ok = ok && arrived() && __all_sync(0xffffffffu, mbar_wait_bounded(p_full, (uint32_t)(t & 1)));
            if (!ok) break;
            pg_fence_after();
            if (pg_elect()) {
                const uint64_t dv = pat_v_desc(ring + (it % PAT_SLOTS) * PAT_TILE_BYTES);
#pragma unroll
                for (int k = 0; k < 4; k++) {   // 16 keys: 2048 bytes of V, eight columns of probabilities on
                    pat_mma_ta(t_o, t_ph + 8u * k, dv + (uint64_t)(k * (2048 >> 4)), PAT_IDESC_O, (t | k) != 0);
                    pat_mma_ta(t_o, t_pl + 8u * k, dv + (uint64_t)(k * (2048 >> 4)), PAT_IDESC_O, 1u);
                }
                pg_commit(&empty[it % PAT_SLOTS]);
                pg_commit(pv_done);
            }
            __syncwarp();
            it++;
        }
    } else if (lane == 0) {
        uint32_t it = 0;
        auto copy = [&](const PgTensorMap *map, int t) {
            const uint32_t s = it % PAT_SLOTS, dst = smem + PAT_Q_BYTES + s * PAT_TILE_BYTES;
            ok = ok && mbar_wait_bounded(&empty[s], ((it / PAT_SLOTS) & 1u) ^ 1u);
            if (!ok) return;
            mbar_arrive_expect_tx(&full[s], PAT_TILE_BYTES);
            pg_tma_2d(dst, map, kv_h * HD, t * PAT_KEYS, &full[s]);
            pg_tma_2d(dst + PAT_KEYS * 128, map, kv_h * HD + 64, t * PAT_KEYS, &full[s]);
            it++;
        };
        if (n_tiles > 0) copy(&maps.k, 0);
        for (int t = 0; t < n_tiles && ok; t++) {
            if (t + 1 < n_tiles) copy(&maps.k, t + 1);
            copy(&maps.v, t);
        }
        pg_drain(full, it, PAT_SLOTS);
    }
    if (!ok) *s_failed = 1;
    __syncwarp();
    pg_fence_before();
    __syncthreads();
    if (warp == 4) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
        if (lane == 0 && *s_failed && err_flag) atomicExch(err_flag, DEV_ERR_GEMM_TIMEOUT);
    }
}

}  // namespace rnb
