// Prefill matmul of short rows (less than four blocks) for up to 128 tokens: the product of prefill_gemm_pair.cuh with two CTAs
// of one SM each instead of a pair, weights dequantised into shared memory.  And what the cut kernels share: the sum over a cluster.
//
// A CTA owns 128 weight rows x all tokens.  A stage is 64 elements of K: nt tokens x 128 bytes by one tiled TMA copy, and 128 weight
// rows that eight warps dequantise straight into the operand tile (layouts as in prefill_gemm.cuh).  Weights do not depend on the
// previous launch: the CTA asks L2 for its rows and dequantises its first stages before the dependency wait; only the token
// copies and the stores come after it.  Warps 0-7 dequantise, then store; warp 8 issues the MMAs, warp 9 the token copies.  Every
// wait is bounded; after a timeout all threads still meet at the last barriers.
//
// What bounds it: fill and drain of a launch of four to twelve stages.
#pragma once
#include "prefill_gemm.cuh"

namespace rnb {

constexpr int PS_THREADS = 320;
constexpr int PS_MAX_STAGES = 5;
constexpr uint32_t PS_SMEM_STAGES = 96 * 1024;   // operand stages; the reduction reuses them: 64 KB of slots, 32 KB of exchange
constexpr size_t PS_SMEM = PS_SMEM_STAGES + 1024;
constexpr int PS_MAX_KS = 8;

struct PsParams {
    int seq, cols, nt, stages;   // nt: tokens, rounded up to a multiple of 16
    uint32_t tmem_cols;
};

__device__ __forceinline__ void ps_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
template <int N>
__device__ __forceinline__ void ps_tmem_ld(uint32_t taddr, uint32_t (&v)[N]) {
    static_assert(N == 8 || N == 16, "columns per load");
    if constexpr (N == 16)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                       "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                     : "r"(taddr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                     : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Adds the accumulators of a cluster's ks CTAs (one: its own).  A round gives every CTA up to ps_per_round chunks of
// SUB * GROUPS tokens: the others send it theirs of those chunks, it adds them in rank order with its own and calls
// f(chunk, count, sums).  Two cluster barriers a round, so few rounds: one or two at 256 tokens.  A worker warp holds the rows of
// lane quarter q and a chunk's tokens group * SUB ..; all threads of the CTA come through here.  `smem` takes BYTES for the
// accumulators that arrive, four tokens of a row at a time (one at a time: 203 tokens of 4096 x 14336 over three pairs 56 -> 51 us).  CTA r
// of the sum is CTA step * r + first of the cluster.
constexpr uint32_t PS_SLOT_BYTES = 64 * 1024;
__host__ __device__ inline int ps_per_round(int ks, uint32_t slot, uint32_t bytes = PS_SLOT_BYTES) { return ks > 1 ? (int)(bytes / slot) / (ks - 1) : 1; }
template <int SUB, int GROUPS, uint32_t BYTES = PS_SLOT_BYTES, class F>
__device__ __forceinline__ void ps_reduce(int ks, int kr, int n_chunks, uint8_t *smem, uint32_t tmem, bool worker, int q, int group, bool fin, F &&f,
                                          int step = 1, int first = 0) {
    constexpr int CT = SUB * GROUPS;                  // tokens per chunk
    constexpr uint32_t SLOT = CT * PG_ROWS * 4;       // one CTA's accumulators of a chunk: [four tokens][row][token]
    static_assert((PS_MAX_KS / 2 - 1) * SLOT <= BYTES, "a slot per sender");
    const int lane = threadIdx.x & 31, M = ps_per_round(ks, SLOT, BYTES);
    const uint32_t base = smem_u32(smem), mine = (uint32_t)(group * SUB * PG_ROWS + (q * 32 + lane) * 4) * 4u;
    const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(group * SUB);
    int count = 0;
    for (int c0 = 0; c0 < n_chunks; c0 += M * ks) {
        if (ks > 1) {
            if (c0 > 0) ps_cluster_sync();   // the slots are free again
            if (worker)
                for (int i = 1; i < ks; i++) {
                    const int to = (kr + i) % ks;
                    for (int m = 0; m < M; m++) {
                        const int cc = c0 + m * ks + to;
                        if (cc >= n_chunks) break;
                        uint32_t v[SUB];
                        if (fin) ps_tmem_ld<SUB>(lanes + (uint32_t)(cc * CT), v);
                        const uint32_t dst = ps_map(base + (uint32_t)((kr < to ? kr : kr - 1) * M + m) * SLOT + mine, step * to + first);
#pragma unroll
                        for (int t = 0; t < SUB; t += 4)
                            ps_st_remote4(dst + (uint32_t)(t * PG_ROWS * 4), fin ? v[t] : 0u, fin ? v[t + 1] : 0u, fin ? v[t + 2] : 0u, fin ? v[t + 3] : 0u);
                    }
                }
            ps_cluster_sync();
        }
        for (int m = 0; m < M; m++) {
            const int cc = c0 + m * ks + kr;
            if (!worker || cc >= n_chunks) break;
            uint32_t v[SUB];
            if (fin) ps_tmem_ld<SUB>(lanes + (uint32_t)(cc * CT), v);
            float s[SUB];
#pragma unroll
            for (int t = 0; t < SUB; t += 4) {
                const uint8_t *part = smem + (size_t)m * SLOT + mine + t * PG_ROWS * 4;
                for (int r = 0; r < ks; r++) {
                    const float4 a = r == kr ? fin ? make_float4(__uint_as_float(v[t]), __uint_as_float(v[t + 1]), __uint_as_float(v[t + 2]), __uint_as_float(v[t + 3]))
                                                   : make_float4(0.f, 0.f, 0.f, 0.f)
                                             : *reinterpret_cast<const float4 *>(part + (size_t)(r < kr ? r : r - 1) * M * SLOT);
                    s[t] = r ? s[t] + a.x : a.x, s[t + 1] = r ? s[t + 1] + a.y : a.y, s[t + 2] = r ? s[t + 2] + a.z : a.z, s[t + 3] = r ? s[t + 3] + a.w : a.w;
                }
            }
            f(cc, count++, s);
        }
    }
}

// Stores a tile with eight worker warps: warp w holds tokens (w >> 2) * SUB .. of a chunk.
template <int SUB>
__device__ __forceinline__ void ps_finish(const PgJob &job, const PsParams &P, uint8_t *smem, uint32_t tmem, int n0, bool fin) {
    constexpr int CT = 2 * SUB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = warp & 3, sub = (warp >> 2) & 1, rows = job.rows;
    const int end = P.seq, n_chunks = (end + CT - 1) / CT;
    float *ex = reinterpret_cast<float *>(smem + PS_SLOT_BYTES);   // gate / up exchange, two buffers in turn
    const bool pair = job.w2 != nullptr;
    ps_reduce<SUB, 2>(1, 0, n_chunks, smem, tmem, warp < 8, q, sub, fin, [&](int cc, int j, const float (&s)[SUB]) {
        const int tok0 = cc * CT;
        if (pair) {
            // gate rows on lane quarters 0 and 1, the same rows of up on 2 and 3: each warp finishes half of its tokens
            float *buf = ex + (size_t)(j & 1) * (CT * PG_ROWS);
#pragma unroll
            for (int t = 0; t < SUB; t++) buf[(sub * SUB + t) * PG_ROWS + q * 32 + lane] = s[t];
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const int row = n0 + (q & 1) * 32 + lane, t_lo = sub * SUB + (q >> 1) * (SUB / 2);
            if (fin && row < rows) {
#pragma unroll
                for (int t = t_lo; t < t_lo + SUB / 2; t++) {
                    const float g = buf[t * PG_ROWS + (q & 1) * 32 + lane], u = buf[t * PG_ROWS + 64 + (q & 1) * 32 + lane];
                    // fast exponential and division: their 2^-21 relative error disappears in the bf16 rounding below
                    const float a = __fdividef(g, 1.0f + __expf(-g)) * u;
                    if (tok0 + t < end) job.yb[(size_t)(tok0 + t) * rows + row] = (uint16_t)(pg_pack_bf16(a, 0.f) & 0xffffu);
                }
            }
        } else if (fin && n0 + q * 32 + lane < rows) {
            float *dst = job.y + (size_t)(tok0 + sub * SUB) * rows + n0 + q * 32 + lane;
#pragma unroll
            for (int t = 0; t < SUB; t++)
                if (tok0 + sub * SUB + t < end) dst[(size_t)t * rows] = s[t];
        }
    });
}

// grid = row tiles of all jobs; 320 threads; dynamic shared memory PS_SMEM.
RNB_GLOBAL void __launch_bounds__(PS_THREADS, 2)
prefill_gemm_split_kernel(const __grid_constant__ PgJobs jobs, const __grid_constant__ PgTensorMap tmap_x, const PsParams P, int *err_flag) {
    extern __shared__ __align__(1024) uint8_t pg_smem_raw[];
    __shared__ __align__(8) uint64_t full[PS_MAX_STAGES], empty[PS_MAX_STAGES], done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    pdl_launch_dependents();
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(pg_smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = (int)blockIdx.x;
    int jsel = 0;
    for (int i = 1; i < jobs.n; i++)
        if (tile >= jobs.j[i].tile0) jsel = i;
    const PgJob &job = jobs.j[jsel];
    const int rows = job.rows, S = P.stages;
    const bool pair = job.w2 != nullptr, q4 = job.type == TYPE_Q4_K;
    const uint32_t BLK = q4 ? Q4K_BYTES : Q6K_BYTES, x_bytes = (uint32_t)P.nt * 128u, stage_bytes = x_bytes + PG_B_BYTES;
    const int n0 = (tile - job.tile0) * (pair ? PG_ROWS / 2 : PG_ROWS);
    const int nb = P.cols >> 8, KT = nb * 4;
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 9);    // one arrival per dequantising warp + the thread that issues the token copies
            mbar_init(&empty[s], 1);   // tcgen05.commit
        }
        mbar_init(&done_bar, 1);
        mbar_fence_init();
        s_failed = 0;
    }
    __syncthreads();
    bool ok = true;

    if (warp < 8) {
        const int row = tid >> 1, h = tid & 1, rr = row & 7;
        const size_t rb = (size_t)nb * BLK;
        // rows past the end repeat the last one (never stored)
        const uint8_t *wr = (pair ? (row < PG_ROWS / 2 ? job.w : job.w2) + (size_t)min(n0 + (row & (PG_ROWS / 2 - 1)), rows - 1) * rb
                                  : job.w + (size_t)min(n0 + row, rows - 1) * rb);
        for (uint32_t o = 128u * (uint32_t)h; o < (uint32_t)nb * BLK; o += 256u) asm volatile("prefetch.global.L2 [%0];" ::"l"(wr + o));
        uint8_t *const brow = smem + x_bytes + (row >> 3) * 1024 + rr * 128;
        int s = 0;
        uint32_t phase = 0;
        auto begin = [&]() { return __all_sync(0xffffffffu, mbar_wait_bounded(&empty[s], phase ^ 1u)); };   // warp-uniform: shuffles follow
        auto end = [&]() {
            pg_proxy_fence();
            __syncwarp();
            if (lane == 0) pg_arrive(&full[s]);
            if (++s == S) s = 0, phase ^= 1u;
        };
        if (q4) {
            // a whole block (four stages) is fetched while the one before it is used
            uint2 hh, hn = make_uint2(0u, 0u);
            uint4 qc[4], qn[4];
            auto load = [&](const uint8_t *blk, uint2 &hd, uint4 (&qq)[4]) {
                hd = ldg_nc_u2(blk + 8 * h);
#pragma unroll
                for (int g = 0; g < 4; g++) qq[g] = ldg_nc_u4(blk + 16 + 32 * g + 16 * h);
            };
            load(wr, hh, qc);
            for (int b = 0; b < nb && ok; b++) {
                wr += BLK;
                if (b + 1 < nb) load(wr, hn, qn);
                const uint32_t ox = __shfl_xor_sync(0xffffffffu, hh.x, 1), oy = __shfl_xor_sync(0xffffffffu, hh.y, 1);
                const uint4 hdr = h ? make_uint4(ox, oy, hh.x, hh.y) : make_uint4(hh.x, hh.y, ox, oy);
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    if (ok) ok = begin();
                    if (!ok) break;
                    const uint4 other = pg_pair_exchange(qc[g]);
                    pg_dequant_q4(hdr, h ? other : qc[g], h ? qc[g] : other, g, h, brow + (uint32_t)s * stage_bytes, rr);
                    end();
                }
                hh = hn;
#pragma unroll
                for (int g = 0; g < 4; g++) qc[g] = qn[g];
            }
        } else {
            PgRawQ6 cur, nxt;
            pg_load_q6(cur, wr, 0, h);
            for (int hb = 0; hb < 2 * nb && ok; hb++) {   // half blocks of 128 elements, two stages each
                if (hb + 1 < 2 * nb) pg_load_q6(nxt, wr + (size_t)((hb + 1) >> 1) * BLK, (hb + 1) & 1, h);
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    if (ok) ok = begin();
                    if (!ok) break;
                    pg_dequant_q6(cur, g, h, brow + (uint32_t)s * stage_bytes, rr);
                    end();
                }
                cur = nxt;
            }
        }
    } else if (warp == 8) {
        pdl_wait();   // tensor memory is asked for when no earlier launch can still hold it
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(P.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        __syncwarp();
        const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(P.nt >> 3) << 17) | ((uint32_t)(PG_ROWS >> 4) << 24);
        int s = 0;
        uint32_t phase = 0;
        for (int kt = 0; kt < KT && ok; kt++) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[s], phase));
            if (!ok) break;
            pg_fence_after();
            if (pg_elect()) {
                const uint32_t x_addr = smem_u32(smem + (uint32_t)s * stage_bytes);
                const uint64_t dx = pg_smem_desc(x_addr), dw = pg_smem_desc(x_addr + x_bytes);
#pragma unroll
                for (int k = 0; k < 4; k++) ps_mma(tmem, dw + 2u * k, dx + 2u * k, idesc, (kt > 0 || k > 0) ? 1u : 0u);   // 32 bytes on
                pg_commit(&empty[s]);
            }
            __syncwarp();
            if (++s == S) s = 0, phase ^= 1u;
        }
        if (ok && pg_elect()) pg_commit(&done_bar);
        __syncwarp();
    } else if (lane == 0) {
        pdl_wait();   // the tokens are the previous launch's result
        int s = 0, issued = 0;
        uint32_t phase = 0;
        for (int kt = 0; kt < KT && ok; kt++) {
            ok = mbar_wait_bounded(&empty[s], phase ^ 1u);
            if (!ok) break;
            mbar_arrive_expect_tx(&full[s], x_bytes);
            pg_tma_2d(smem_u32(smem + (uint32_t)s * stage_bytes), &tmap_x, kt * PG_K, 0, &full[s]);
            issued = kt + 1;
            if (++s == S) s = 0, phase ^= 1u;
        }
        pg_drain(full, (uint32_t)issued, (uint32_t)S);   // the stages are reused
    }
    if (!ok) s_failed = 1;
    __syncthreads();   // the accumulators' address; a failure of any role
    pdl_wait();        // every thread that stores comes after the launches before this one
    bool fin = s_failed == 0;
    fin = __all_sync(0xffffffffu, fin && mbar_wait_bounded(&done_bar, 0u));
    if (!fin) s_failed = 1;
    pg_fence_after();
    const uint32_t tmem = tmem_slot;
    ps_finish<16>(job, P, smem, tmem, n0, fin);
    pg_fence_before();
    __syncthreads();
    if (warp == 8) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P.tmem_cols) : "memory");
        if (lane == 0 && s_failed && err_flag) atomicExch(err_flag, DEV_ERR_GEMM_TIMEOUT);
    }
}

}  // namespace rnb
