// Prefill matmul on pairs of SMs with tiles of up to 512 tokens: the product of prefill_gemm_pair.cuh with the weights dequantised into
// shared memory, so that accumulators take all of tensor memory.  For prompts whose 512-token tiles fill the chip in one round while
// narrower ones need two: each weight is dequantised once (4096 x 14336 Q6_K, 2048 tokens: 153 us, 200 with 256-token tiles).
//
// A pair of CTAs (a cluster of two) multiplies 256 weight rows x up to 512 tokens: each CTA dequantises its own 128 rows,
// brings in half of the tokens, and holds its rows' accumulators in all 512 columns of its tensor memory (two token parts
// of n1 and n2 columns).
//
// Blocks of 256 elements of the 128 rows come into shared memory as they are, by tiled copies, one block ahead: the
// dequantising warps fence their stores for the tensor pipe at every stage, and that fence also waits for loads from
// global memory that are still under way.
//
// Persistent: a pair walks its tiles (token tiles fastest, so that a weight row crosses DRAM once).  Warps 0-15
// dequantise, two groups of eight that take two of a block's four stages each; behind the first stage of the next tile
// they write the finished tile from tensor memory and hand the columns back.  Warp 16 of the even CTA issues the MMAs,
// warp 17 of each CTA its token copies, warp 18 those of the weights.  A stage fills on each CTA's own barrier; warp 16 of
// the odd CTA waits for its own and passes one arrival on to the even CTA's: a release and an acquire across the cluster
// stand between what the odd CTA wrote and the MMA that reads it, and the dequantising warps do not wait for them.
// A commit reaches both CTAs.  Every wait is bounded; after a timeout all threads still meet at the cluster barrier.
//
// What bounds it: the dequantising warps' chain of a stage (fences, hand-over), 2.5 us a block of 256 elements up to 450 tokens.
#pragma once
#include "prefill_gemm_pair.cuh"

namespace rnb {

constexpr int PW_STAGES = 4;       // one block of K
constexpr int PW_WORKERS = 16;     // dequantising warps
constexpr int PW_THREADS = (PW_WORKERS + 3) * 32;
constexpr int PW_TOK = 512;
constexpr uint32_t PW_RING = PW_STAGES * (PW_TOK / 2 * 128 + PG_B_BYTES);
constexpr size_t PW_SMEM = PW_RING + PT_RAW_BYTES + 1024;

struct PwParams {
    int seq, cols, n1, n2;             // n1, n2: tokens of the two parts of a tile (multiples of 32, at most 256)
    int row_tiles, token_tiles, tiles; // tiles: pairs of row tiles x token tiles
    int direct;                        // bit i: job i's rows cannot be described for tiled copies (Q6_K, 2-byte aligned)
};
struct PwMaps {   // tokens of the two parts (boxes of n1 / 2 and n2 / 2), blocks of each job's rows (boxes of 64), of the second matrix of a pair
    PgTensorMap xa, xb, w[PG_MAX_JOBS], w2;
};

// grid = 2 x pairs, cluster (2, 1, 1); PW_THREADS threads; dynamic shared memory PW_SMEM.
RNB_GLOBAL void __launch_bounds__(PW_THREADS, 1)
prefill_gemm_wide_kernel(const __grid_constant__ PgJobs jobs, const __grid_constant__ PwMaps maps, const PwParams P, int *err_flag) {
    extern __shared__ __align__(1024) uint8_t pg_smem_raw[];
    __shared__ __align__(8) uint64_t full[PW_STAGES], empty[PW_STAGES], raw_full, raw_empty, acc_full, acc_free;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    pdl_launch_dependents();
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(pg_smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)blockIdx.x & 1, pair0 = (int)blockIdx.x >> 1, n_pairs = (int)gridDim.x >> 1;
    const int nb = P.cols >> 8, nt = P.n1 + P.n2;
    const uint32_t tok_bytes = (uint32_t)(nt / 2) * 128u, stage_bytes = tok_bytes + PG_B_BYTES;
    if (tid == 0) {
        for (int s = 0; s < PW_STAGES; s++) {
            mbar_init(&full[s], PW_WORKERS / 2 + 1 + (rank == 0));   // the warps of a group + the thread that announces the token copies + the odd CTA
            mbar_init(&empty[s], 1);                                 // tcgen05.commit
        }
        mbar_init(&raw_full, 1);
        mbar_init(&raw_empty, PW_WORKERS);
        mbar_init(&acc_full, 1);
        mbar_init(&acc_free, 2 * PW_WORKERS);
        mbar_fence_init();
        s_failed = 0;
    }
    if (warp == PW_WORKERS) {
        // no launch that holds tensor memory can share an SM with this much shared memory
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pg_fence_before();
    __syncthreads();
    ps_cluster_sync();   // barriers and tensor memory of both CTAs stand
    pg_fence_after();
    const uint32_t tmem = tmem_slot;
    auto job_of = [&](int tile, int &local) {
        const int rt = min(2 * (tile / P.token_tiles) + rank, P.row_tiles - 1);
        int js = 0;
        for (int i = 1; i < jobs.n; i++)
            if (rt >= jobs.j[i].tile0) js = i;
        local = rt - jobs.j[js].tile0;
        return js;
    };
    bool ok = true;

    if (warp < PW_WORKERS) {
        const int grp = warp >> 3, row = (tid & 255) >> 1, h = tid & 1, rr = row & 7;
        uint8_t *const brow = smem + tok_bytes + (row >> 3) * 1024 + rr * 128;
        uint32_t uses = 0, raws = 0;   // blocks that have gone through the ring of stages, of raw blocks
        // a stage: wait for its slot (warp-uniform: shuffles follow), then hand it over
        auto begin = [&](int i) { return __all_sync(0xffffffffu, mbar_wait_bounded(&empty[2 * grp + i], (uses & 1u) ^ 1u)); };
        auto end = [&](int i) {
            pg_proxy_fence();
            __syncwarp();
            if (lane == 0) pg_arrive(&full[2 * grp + i]);
        };
        uint8_t *const dst[2] = {brow + (uint32_t)(2 * grp) * stage_bytes, brow + (uint32_t)(2 * grp + 1) * stage_bytes};
        // tile `tile`, the pair's `count`-th: tensor memory lane = weight row, a warp takes every fourth group of 32 tokens
        auto finish = [&](int tile, int count) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&acc_full, (uint32_t)(count & 1)));
            if (!ok) return;
            pg_fence_after();
            int local;
            const PgJob &job = jobs.j[job_of(tile, local)];
            const bool mine = 2 * (tile / P.token_tiles) + rank < P.row_tiles, pair = job.w2 != nullptr;
            const int q = warp & 3, m0 = (tile % P.token_tiles) * nt, rows = job.rows;
            for (int c = warp >> 2; c < nt / 32; c += 4) {
                const int col = c * 32 < P.n1 ? c * 32 : 256 + c * 32 - P.n1, tok0 = m0 + c * 32;
                if (tok0 >= P.seq) break;
                uint32_t v[32];
                pg_tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)col, v);
                if (!mine) continue;
                if (pair) {
                    // gate rows on even lanes, the same rows of up on odd ones: the lanes of a row finish a token each
                    const int r = local * (PG_ROWS / 2) + q * 16 + (lane >> 1), odd = lane & 1;
                    uint16_t *dst = job.yb + (size_t)(tok0 + odd) * rows + r;
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const float own = __uint_as_float(odd ? v[j + 1] : v[j]);
                        const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, odd ? v[j] : v[j + 1], 1));
                        const float g = odd ? other : own, u = odd ? own : other;
                        // fast exponential and division: their 2^-21 relative error disappears in the bf16 rounding below
                        const float a = __fdividef(g, 1.0f + __expf(-g)) * u;
                        if (r < rows && tok0 + odd + j < P.seq) dst[(size_t)j * rows] = (uint16_t)(pg_pack_bf16(a, 0.f) & 0xffffu);
                    }
                } else {
                    const int r = local * PG_ROWS + q * 32 + lane;
                    float *dst = job.y + (size_t)tok0 * rows + r;
                    if (r < rows) {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (tok0 + j < P.seq) dst[(size_t)j * rows] = __uint_as_float(v[j]);
                    }
                }
            }
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pt_arrive(ps_map(smem_u32(&acc_free), 0));
        };
        // The blocks of this thread's row of the pair's `count`-th tile: group `grp` dequantises stages 2 grp and 2 grp + 1 of
        // each.  The tile before it is finished behind the first stage: the even CTA's MMAs of this one wait for its columns.
        auto blocks = [&](int tile, int count) {
            int local;
            const int js = job_of(tile, local);
            const PgJob &job = jobs.j[js];
            const bool q4 = job.type == TYPE_Q4_K, direct = (P.direct >> js) & 1;
            // gate and up rows alternate
            const uint8_t *const raw = smem + PW_RING + (uint32_t)(job.w2 ? (row & 1) * (PG_ROWS / 2) + (row >> 1) : row) * (q4 ? PT_Q4_PITCH : PT_Q6_PITCH);
            for (int b = 0; b < nb && ok; b++) {
                PgRawQ6 cur;
                uint32_t ql[8], qh[8], sc[2];   // Q4_K: the low and high half of `qs` of the two stages
                uint4 hdr;
                float d = 0.f;
                if (direct) {
                    // rows past the end repeat the last one (never stored)
                    const uint8_t *wr = job.w2 ? (row & 1 ? job.w2 : job.w) + (size_t)min(local * (PG_ROWS / 2) + (row >> 1), job.rows - 1) * nb * Q6K_BYTES
                                               : job.w + (size_t)min(local * PG_ROWS + row, job.rows - 1) * nb * Q6K_BYTES;
                    pg_load_q6(cur, wr + (size_t)b * Q6K_BYTES, grp, h);
                } else {
                    // the block's bytes into registers, and the buffer is free for the next one
                    ok = __all_sync(0xffffffffu, mbar_wait_bounded(&raw_full, raws & 1u));
                    if (!ok) break;
                    raws++;
                    if (q4) {
                        hdr = *reinterpret_cast<const uint4 *>(raw);
#pragma unroll
                        for (int j = 0; j < 2; j++) {
                            *reinterpret_cast<uint4 *>(ql + 4 * j) = *reinterpret_cast<const uint4 *>(raw + 16 + 64 * grp + 16 * j);
                            *reinterpret_cast<uint4 *>(qh + 4 * j) = *reinterpret_cast<const uint4 *>(raw + 48 + 64 * grp + 16 * j);
                        }
                    } else {
                        const uint8_t *const q = raw + (((uint32_t)b * Q6K_BYTES) & 15u);
                        pg_ldg_window<8, 3, true>(q + 64 * grp + 32 * h, ql);
                        pg_ldg_window<8, 3, true>(q + 128 + 32 * grp, qh);
                        d = f16_bits_to_f32(*reinterpret_cast<const uint16_t *>(q + 208));
#pragma unroll
                        for (int i = 0; i < 2; i++) sc[i] = *reinterpret_cast<const uint16_t *>(q + 192 + 8 * grp + 4 * i + 2 * h);
                    }
                    __syncwarp();
                    if (lane == 0) pg_arrive(&raw_empty);
                }
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    ok = ok && begin(i);
                    if (!ok) break;
                    if (q4) {
                        const uint32_t(&q)[8] = i ? qh : ql;
                        pg_dequant_q4(hdr, make_uint4(q[0], q[1], q[2], q[3]), make_uint4(q[4], q[5], q[6], q[7]), 2 * grp + i, h, dst[i], rr);
                    } else if (direct)
                        pg_dequant_q6(cur, i, h, dst[i], rr);
                    else
                        pg_dequant_q6_half(ql, qh, sc[i], d, i == 1, h, dst[i], rr);
                    end(i);
                    if (i == 0 && b == 0 && count > 0) {
                        pdl_wait();   // stores come after the launches before this one
                        finish(tile - n_pairs, count - 1);
                    }
                }
                uses++;
            }
        };
        int count = 0;
        for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs, count++) blocks(tile, count);
        if (count > 0 && ok) {
            pdl_wait();
            finish(pair0 + (count - 1) * n_pairs, count - 1);
        }
    } else if (warp == PW_WORKERS) {
        if (rank == 0) {
            const uint32_t id1 = pt_idesc(P.n1), id2 = pt_idesc(P.n2);
            uint32_t s = 0, phase = 0;
            int count = 0;
            for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs, count++) {
                if (count > 0) ok = __all_sync(0xffffffffu, pt_wait(&acc_free, (uint32_t)((count - 1) & 1)));
                for (int kt = 0; kt < 4 * nb && ok; kt++) {
                    ok = __all_sync(0xffffffffu, pt_wait_shared(&full[s], phase));
                    if (!ok) break;
                    pg_fence_after();
                    if (pg_elect()) {
                        const uint32_t x1 = smem_u32(smem + s * stage_bytes);
                        const uint64_t dx1 = pg_smem_desc(x1), dx2 = pg_smem_desc(x1 + (uint32_t)(P.n1 / 2) * 128u), dw = pg_smem_desc(x1 + tok_bytes);
#pragma unroll
                        for (int k = 0; k < 4; k++) pt_mma(tmem, dw + 2u * k, dx1 + 2u * k, id1, (kt | k) != 0);   // 32 bytes on
#pragma unroll
                        for (int k = 0; k < 4; k++) pt_mma(tmem + 256u, dw + 2u * k, dx2 + 2u * k, id2, (kt | k) != 0);
                        pt_commit(&empty[s]);
                    }
                    __syncwarp();
                    if (++s == PW_STAGES) s = 0, phase ^= 1u;
                }
                if (ok && pg_elect()) pt_commit(&acc_full);
                __syncwarp();
            }
        } else if (lane == 0) {
            uint32_t st = 0;
            for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs)
                for (int kt = 0; kt < 4 * nb && ok; kt++, st++) {
                    const uint32_t s = st % PW_STAGES;
                    ok = mbar_wait_bounded(&full[s], (st / PW_STAGES) & 1u);
                    if (ok) pt_arrive_shared(ps_map(smem_u32(&full[s]), 0));
                }
        }
    } else if (warp == PW_WORKERS + 1) {
        if (lane == 0) {
            pdl_wait();   // the tokens are the previous launch's result
            uint32_t st = 0;
            for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs) {
                const int m0 = (tile % P.token_tiles) * nt;
                for (int kt = 0; kt < 4 * nb && ok; kt++) {
                    const uint32_t s = st % PW_STAGES;
                    ok = mbar_wait_bounded(&empty[s], ((st / PW_STAGES) & 1u) ^ 1u);
                    if (!ok) break;
                    const uint32_t to = smem_u32(smem + s * stage_bytes);
                    mbar_arrive_expect_tx(&full[s], tok_bytes);
                    pg_tma_2d(to, &maps.xa, kt * PG_K, m0 + rank * (P.n1 / 2), &full[s]);
                    pg_tma_2d(to + (uint32_t)(P.n1 / 2) * 128u, &maps.xb, kt * PG_K, m0 + P.n1 + rank * (P.n2 / 2), &full[s]);
                    st++;
                }
            }
            pg_drain(full, st, PW_STAGES);
        }
    } else if (lane == 0) {
        // blocks of K as they are in memory: 64 rows a copy
        uint32_t raws = 0;
        for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs) {
            int local;
            const int js = job_of(tile, local);
            if ((P.direct >> js) & 1) continue;
            const PgJob &job = jobs.j[js];
            const bool q4 = job.type == TYPE_Q4_K;
            const uint32_t pitch = q4 ? PT_Q4_PITCH : PT_Q6_PITCH, to = smem_u32(smem + PW_RING);
            const int y = local * (job.w2 ? PG_ROWS / 2 : PG_ROWS);
            for (int b = 0; b < nb && ok; b++, raws++) {
                ok = mbar_wait_bounded(&raw_empty, (raws & 1u) ^ 1u);
                if (!ok) break;
                const int x = q4 ? b * (int)(Q4K_BYTES / 8) : ((b * (int)Q6K_BYTES) & ~15) / 8;   // 8-byte words, even: a 16-byte boundary
                mbar_arrive_expect_tx(&raw_full, PG_ROWS * pitch);
                pg_tma_2d(to, &maps.w[js], x, y, &raw_full);
                pg_tma_2d(to + PG_ROWS / 2 * pitch, job.w2 ? &maps.w2 : &maps.w[js], x, job.w2 ? y : y + PG_ROWS / 2, &raw_full);
            }
        }
        pg_drain(&raw_full, raws, 1);
    }
    if (!ok) s_failed = 1;
    __syncwarp();
    pg_fence_before();
    __syncthreads();
    ps_cluster_sync();   // the other CTA's memory and barriers are no longer used
    if (warp == PW_WORKERS) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
        if (lane == 0 && s_failed && err_flag) atomicExch(err_flag, DEV_ERR_GEMM_TIMEOUT);
    }
}

}  // namespace rnb
