// Causal softmax attention of a prompt's queries (causal_attention.cuh) on the 5th-generation tensor cores: keys of 128 or
// 192 elements, values of 128, rows that tiled copies can describe and a key ring that has not wrapped yet.
//
// The design of prefill_attention_tiled.cuh: 128 queries of a head per CTA, tiles of 64 keys, a row per thread of warps 0-3, scores,
// output and probabilities in tensor memory, the scores of the next tile under way during the softmax, the output scaled only
// when a maximum has grown by more than 2^8.  Queries and keys are bf16 as they are; probabilities enter as bf16 hi + lo.  A key's
// panels of 64 elements come from its head's rows and from the rows that all heads share.  Two CTAs per SM (at most 112 KB,
// 256 tensor-memory columns each).  Every wait is bounded.
//
// What bounds it: the softmax warps, as there.  Whole prompts, together with the matmul of pairs: four Punisun layers of 8B
// widths at 2048 tokens 5.27 -> 5.12 ms, three Dutivik layers at 1999 tokens 4.33 -> 4.16 ms.
#pragma once
#include "causal_attention.cuh"
#include "prefill_attention_tiled.cuh"

namespace rnb {

struct CausalAttentionMaps {
    PgTensorMap q, k, k2, v;   // boxes of 64 columns x 128 (queries) or 64 rows
};
constexpr uint32_t CT_PANEL_Q = CA_ROWS * 128, CT_PANEL_K = CA_KEYS * 128, CT_V_BYTES = CA_KEYS * 256;
constexpr int ct_v_slots(int kp) { return kp == 2 ? 2 : 1; }
constexpr uint32_t ct_tiles(int kp) { return (uint32_t)kp * CT_PANEL_Q + 2u * (uint32_t)kp * CT_PANEL_K + (uint32_t)ct_v_slots(kp) * CT_V_BYTES; }
constexpr size_t ct_smem(int kp) { return ct_tiles(kp) + 128; }   // + barriers; two CTAs per SM leave no room to align
// D = f32, A = B = bf16, M = 128
constexpr uint32_t CT_IDESC_S = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(CA_KEYS >> 3) << 17) | ((uint32_t)(CA_ROWS >> 4) << 24);
constexpr uint32_t CT_IDESC_O = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(CA_ROWS >> 4) << 24);   // values dims-major

// grid = (heads, ceil(tokens / 128)), PAT_THREADS threads.  KP: panels of 64 elements of a key; pos0: the first query's position.
template <int KP>
RNB_GLOBAL void __launch_bounds__(PAT_THREADS, 2)
causal_attention_tc_kernel(const __grid_constant__ CausalAttentionArgs a, const __grid_constant__ CausalAttentionMaps maps, int pos0, int *err_flag) {
    extern __shared__ __align__(1024) uint8_t ct_mem[];
    constexpr int NV = ct_v_slots(KP);
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.x, hk = h / a.group;
    uint64_t *const bars = reinterpret_cast<uint64_t *>(ct_mem + ct_tiles(KP));
    uint64_t *const kfull = bars, *const kempty = bars + 2, *const vfull = bars + 4, *const vempty = bars + 6, *const q_full = bars + 8, *const s_full = bars + 9,
                    *const s_free = bars + 10, *const p_full = bars + 11, *const pv_done = bars + 12;
    volatile uint32_t *const tmem_slot = reinterpret_cast<volatile uint32_t *>(bars + 13);
    volatile int *const s_failed = reinterpret_cast<volatile int *>(bars + 14);
    const uint32_t smem = smem_u32(ct_mem), k_at = smem + KP * CT_PANEL_Q, v_at = k_at + 2 * KP * CT_PANEL_K;
    const int i0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * CA_ROWS;   // long rows first
    const int kv_len = pos0 + a.tokens;
    const int n_keys = min(kv_len, pos0 + i0 + CA_ROWS), t_end = (n_keys + CA_KEYS - 1) / CA_KEYS;
    const int t_first = a.window > 0 ? max(0, pos0 + i0 - a.window + 1) / CA_KEYS : 0, n_tiles = t_end - t_first;
    if (tid == 0) {
        for (int s = 0; s < 8; s++) mbar_init(&bars[s], 1);
        mbar_init(q_full, 1);
        mbar_init(s_full, 1);
        mbar_init(s_free, 4);
        mbar_init(p_full, 4);
        mbar_init(pv_done, 1);
        mbar_fence_init();
        *s_failed = (smem & 1023u) != 0;
    }
    pdl_wait();   // queries, keys and values are the previous launch's result; tensor memory is asked for when no earlier launch can still hold it
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
        const int qi = i0 + warp * 32 + lane;
        const bool live = qi < a.tokens;
        const int pos = live ? pos0 + qi : kv_len - 1;   // rows past the end see what the last one sees and are never stored
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        const float sl2 = a.scale * 1.4426950408889634f;
        float m_ref = -INFINITY, l_run = 0.f;
        for (int t = 0; t < n_tiles && ok; t++) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(s_full, (uint32_t)(t & 1)));
            if (!ok) break;
            pg_fence_after();
            uint32_t s[CA_KEYS];
            pat_tmem_ld64(t_s + lanes, s);
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pg_arrive(s_free);
            // the tile's keys first .. last are visible
            const int last = pos - (t_first + t) * CA_KEYS, first = a.window > 0 ? last - a.window + 1 : 0;
            if (last < CA_KEYS - 1 || first > 0) {
#pragma unroll
                for (int i = 0; i < CA_KEYS; i++)
                    if (i > last || i < first) s[i] = 0xff800000u;   // -inf
            }
            float mxs[4];
#pragma unroll
            for (int j = 0; j < 4; j++) mxs[j] = __uint_as_float(s[j]);
#pragma unroll
            for (int i = 4; i < CA_KEYS; i++) mxs[i & 3] = fmaxf(mxs[i & 3], __uint_as_float(s[i]));
            const float mx = fmaxf(fmaxf(mxs[0], mxs[1]), fmaxf(mxs[2], mxs[3])) * sl2;   // sl2 > 0
            float corr = 1.0f;
            if (mx > m_ref + PAT_GROWTH || m_ref == -INFINITY) {
                const float m_new = fmaxf(mx, m_ref);
                corr = exp2f(m_ref - (m_new == -INFINITY ? 0.f : m_new));
                m_ref = m_new;
            }
            const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
            const uint64_t sl22 = pg_pair_f32(sl2, sl2), nm2 = pg_pair_f32(-m_use, -m_use);
            uint64_t sum[2] = {0, 0};
            uint32_t ph[32], pl[32];
#pragma unroll
            for (int i = 0; i < 32; i++) {
                const float2 x = pat_fma2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]), sl22, nm2);
                const float p0 = pat_exp2(x.x), p1 = pat_exp2(x.y);
                pat_add2(sum[i & 1], p0, p1);
                lt_split(p0, p1, ph[i], pl[i]);
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
        if (ok && n_tiles > 0) {
            pg_fence_after();
            float inv = a.out_mul / l_run;
            if (a.gate && live) inv /= 1.0f + expf(-a.gate[(size_t)qi * a.ldg + h]);
            __syncwarp();
#pragma unroll 1
            for (int c = 0; c < 4; c++) {
                uint32_t v[32];
                pg_tmem_ld32(t_o + lanes + (uint32_t)c * 32u, v);
                if (!live) continue;
                auto o = [&](int i) { return __uint_as_float(v[i]) * inv; };
#pragma unroll
                for (int i = 0; i < 32; i += 8)
                    *reinterpret_cast<uint4 *>(a.act + (size_t)qi * a.lda + (size_t)h * 128 + c * 32 + i) =
                        make_uint4(pg_pack_bf16(o(i), o(i + 1)), pg_pack_bf16(o(i + 2), o(i + 3)), pg_pack_bf16(o(i + 4), o(i + 5)), pg_pack_bf16(o(i + 6), o(i + 7)));
            }
        }
    } else if (warp == 4) {
        auto scores = [&](int t) {
            ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&kfull[t & 1], (uint32_t)((t >> 1) & 1)));
            if (!ok) return;
            pg_fence_after();
            if (pg_elect()) {
#pragma unroll
                for (int p = 0; p < KP; p++) {
                    const uint64_t dq = pg_smem_desc(smem + (uint32_t)p * CT_PANEL_Q), dk = pg_smem_desc(k_at + (uint32_t)((t & 1) * KP + p) * CT_PANEL_K);
#pragma unroll
                    for (int k = 0; k < 4; k++) ps_mma(t_s, dq + 2u * k, dk + 2u * k, CT_IDESC_S, (p | k) != 0);   // 16 elements, 32 bytes on
                }
                pg_commit(&kempty[t & 1]);
                pg_commit(s_full);
            }
            __syncwarp();
        };
        if (n_tiles > 0) {
            ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(q_full, 0u));
            scores(0);
        }
        for (int t = 0; t < n_tiles && ok; t++) {
            if (t + 1 < n_tiles) {
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(s_free, (uint32_t)(t & 1)));
                scores(t + 1);
            }
            ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&vfull[t % NV], (uint32_t)((t / NV) & 1)) && mbar_wait_bounded(p_full, (uint32_t)(t & 1)));
            if (!ok) break;
            pg_fence_after();
            if (pg_elect()) {
                const uint64_t dv = pat_v_desc(v_at + (uint32_t)(t % NV) * CT_V_BYTES);
#pragma unroll
                for (int k = 0; k < 4; k++) {   // 16 keys: 2048 bytes of the values, eight columns of probabilities on
                    pat_mma_ta(t_o, t_ph + 8u * k, dv + (uint64_t)(k * (2048 >> 4)), CT_IDESC_O, (t | k) != 0);
                    pat_mma_ta(t_o, t_pl + 8u * k, dv + (uint64_t)(k * (2048 >> 4)), CT_IDESC_O, 1u);
                }
                pg_commit(&vempty[t % NV]);
                pg_commit(pv_done);
            }
            __syncwarp();
        }
    } else if (lane == 0 && ok && n_tiles > 0) {
        const int own = a.dim / 64;   // panels from the head's rows; the others are shared by all heads
        int nk = 0, nv = 0;
        auto keys = [&](int t) {
            uint64_t *bar = &kfull[t & 1];
            ok = ok && mbar_wait_bounded(&kempty[t & 1], (uint32_t)(((t >> 1) & 1) ^ 1));
            if (!ok) return;
            mbar_arrive_expect_tx(bar, KP * CT_PANEL_K);
            for (int p = 0; p < KP; p++)
                pg_tma_2d(k_at + (uint32_t)((t & 1) * KP + p) * CT_PANEL_K, p < own ? &maps.k : &maps.k2, p < own ? hk * a.dim + 64 * p : 64 * (p - own), (t_first + t) * CA_KEYS, bar);
            nk++;
        };
        mbar_arrive_expect_tx(q_full, KP * CT_PANEL_Q);
        for (int p = 0; p < KP; p++) pg_tma_2d(smem + (uint32_t)p * CT_PANEL_Q, &maps.q, h * (a.dim + a.dim2) + 64 * p, i0, q_full);
        keys(0);
        for (int t = 0; t < n_tiles && ok; t++) {
            if (t + 1 < n_tiles) keys(t + 1);
            uint64_t *bar = &vfull[t % NV];
            ok = ok && mbar_wait_bounded(&vempty[t % NV], (uint32_t)(((t / NV) & 1) ^ 1));
            if (!ok) break;
            mbar_arrive_expect_tx(bar, CT_V_BYTES);
            for (int p = 0; p < 2; p++) pg_tma_2d(v_at + (uint32_t)(t % NV) * CT_V_BYTES + (uint32_t)p * CT_PANEL_K, &maps.v, hk * 128 + 64 * p, (t_first + t) * CA_KEYS, bar);
            nv++;
        }
        pg_drain(q_full, 1, 1);
        pg_drain(kfull, (uint32_t)nk, 2);
        pg_drain(vfull, (uint32_t)nv, NV);
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
