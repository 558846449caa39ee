// Dense (bf16) weight matrices of the layered decoders: y[t][row] = sum_k W[row][k] * x[t][k].
//
//   dense_gemv_kernel       1..8 tokens, f32 activations: one warp per two rows, weights streamed by
//                           16-byte loads (the first ones issued before the dependency wait)
//   dense_gemm_pair_kernel  many tokens, bf16 activations, tcgen05: 256 rows x up to 512 tokens per pair of SMs
//   dense_gemm_split_kernel the same for prompts whose tiles do not fill the chip: K cut over a cluster
//   dense_gemm_simt_kernel  many tokens in true f32 (and bf16 activations whose rows are not
//                           16-byte aligned, which the tiled copies cannot describe)
//
// All accumulate in f32.  Matrices that go out together share a launch (jobs).  A job with w2 is a
// gate + up pair: the result is act(w x) * (w2 x), act the tanh form of gelu or silu.
#pragma once
#include <cuda_bf16.h>

#include "bounded_walk.hpp"
#include "common.cuh"
#include "prefill_gemm.cuh"
#include "prefill_gemm_pair.cuh"
#include "prefill_gemm_split.cuh"

namespace rnb {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float to_f32(float v) { return v; }
__device__ __forceinline__ float to_f32(bf16 v) { return __bfloat162float(v); }
template <class T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ bf16 from_f32<bf16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float gelu_tanh_f32(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
// The same through 0.5 (1 + tanh a) = 1 / (1 + exp(-2 a)), for results that are rounded to bf16 next: the fast
// exponential's and division's errors (about 2^-21) disappear in that rounding.
__device__ __forceinline__ float gelu_tanh_fast(float z) {
    return __fdividef(z, 1.0f + __expf(-1.5957691216057308f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float silu_f32(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__device__ __forceinline__ float silu_fast(float z) { return __fdividef(z, 1.0f + __expf(-z)); }
constexpr int ACT_GELU_TANH = 0, ACT_SILU = 1;
__device__ __forceinline__ float gate_act(int act, float z) { return act == ACT_SILU ? silu_f32(z) : gelu_tanh_f32(z); }
__device__ __forceinline__ float gate_act_fast(int act, float z) { return act == ACT_SILU ? silu_fast(z) : gelu_tanh_fast(z); }

// A decay in (0, 1) from its projection x: exp(-exp(x)), or sigmoid(x)^inv_tau taken through the logarithm of the sigmoid
// (whose absolute error is what counts for the power).
constexpr int DECAY_EXP = 0, DECAY_SIGMOID_ROOT = 1;
__device__ __forceinline__ float decay_of(int kind, float x, float inv_tau) {
    return kind == DECAY_SIGMOID_ROOT ? expf((fminf(x, 0.f) - logf(1.0f + expf(-fabsf(x)))) * inv_tau) : expf(-expf(x));
}
// sigmoid(x)^inv_tau for tensor-core products, whose operands were rounded to bf16: the fast exponential and logarithm
// (absolute error of the logarithm 2^-21).
__device__ __forceinline__ float sigmoid_root_fast(float x, float inv_tau) {
    return __expf((fminf(x, 0.f) - __logf(1.0f + __expf(-fabsf(x)))) * inv_tau);
}

constexpr int DENSE_MAX_JOBS = 6;

// ---- few tokens ---------------------------------------------------------------------------------
struct DenseVecJob {
    const bf16 *w, *w2;   // [rows][cols]; w2: the up half of a gate + up pair
    const float *x;       // token t at x + t * ldx
    float *y;             // token t at y + t * ldy
    int rows, cols, ldx, ldy, cta0, vec, act;   // vec: rows of 16-byte aligned weights (cols % 8 == 0) and inputs
};
struct DenseVecJobs {
    DenseVecJob j[DENSE_MAX_JOBS];
    int n, ksplit;   // ksplit (1, 2, 4): warps that share a pair of rows, each taking every ksplit-th 1024 columns
};
constexpr int DV_WARPS = 4, DV_UNROLL = 4;

// ksplit warps own two output rows (or the gate and the up row of one output).  T = tokens, 1 .. 8.
template <int T>
RNB_GLOBAL void __launch_bounds__(DV_WARPS * 32)
dense_gemv_kernel(const __grid_constant__ DenseVecJobs jobs) {
    pdl_launch_dependents();
    int js = 0;
    for (int i = 1; i < jobs.n; i++)
        if ((int)blockIdx.x >= jobs.j[i].cta0) js = i;
    const DenseVecJob &job = jobs.j[js];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ks = jobs.ksplit, part = warp & (ks - 1);
    const int unit = ((int)blockIdx.x - job.cta0) * (DV_WARPS / ks) + warp / ks;
    __shared__ float s_part[DV_WARPS][2][T];
    const bool pair = job.w2 != nullptr;
    const int r0 = pair ? unit : 2 * unit, rows = job.rows, cols = job.cols;
    const bool live = r0 < rows, two = pair || r0 + 1 < rows;
    const bf16 *w0 = job.w + (size_t)min(r0, rows - 1) * cols;
    const bf16 *w1 = pair ? job.w2 + (size_t)min(r0, rows - 1) * cols : job.w + (size_t)min(r0 + 1, rows - 1) * cols;
    float a0[T], a1[T];
#pragma unroll
    for (int t = 0; t < T; t++) a0[t] = a1[t] = 0.f;
    if (job.vec) {
        uint4 b0[DV_UNROLL], b1[DV_UNROLL];
        const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
        auto fetch = [&](int k0) {
#pragma unroll
            for (int u = 0; u < DV_UNROLL; u++) {
                const int k = k0 + u * 256 + lane * 8;
                b0[u] = k < cols ? ldg_nc_u4(w0 + k) : z4;
                b1[u] = k < cols ? ldg_nc_u4(w1 + k) : z4;
            }
        };
        const int step = 256 * DV_UNROLL * ks;
        fetch(part * 256 * DV_UNROLL);        // weights do not depend on the previous launch
        pdl_wait();
        for (int k0 = part * 256 * DV_UNROLL; k0 < cols; k0 += step) {
            uint4 c0[DV_UNROLL], c1[DV_UNROLL];
#pragma unroll
            for (int u = 0; u < DV_UNROLL; u++) c0[u] = b0[u], c1[u] = b1[u];
            if (k0 + step < cols) fetch(k0 + step);
#pragma unroll
            for (int u = 0; u < DV_UNROLL; u++) {
                const int k = k0 + u * 256 + lane * 8;
                if (k >= cols) continue;
                const uint32_t p[4] = {c0[u].x, c0[u].y, c0[u].z, c0[u].w}, q[4] = {c1[u].x, c1[u].y, c1[u].z, c1[u].w};
#pragma unroll
                for (int t = 0; t < T; t++) {
                    const float4 xa = *reinterpret_cast<const float4 *>(job.x + (size_t)t * job.ldx + k);
                    const float4 xb = *reinterpret_cast<const float4 *>(job.x + (size_t)t * job.ldx + k + 4);
                    const float xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        a0[t] = fmaf(bf16_lo(p[e]), xv[2 * e], a0[t]);
                        a0[t] = fmaf(bf16_hi(p[e]), xv[2 * e + 1], a0[t]);
                        a1[t] = fmaf(bf16_lo(q[e]), xv[2 * e], a1[t]);
                        a1[t] = fmaf(bf16_hi(q[e]), xv[2 * e + 1], a1[t]);
                    }
                }
            }
        }
    } else {
        pdl_wait();
        for (int k = part * 32 + lane; k < cols; k += 32 * ks) {
            const float p = to_f32(w0[k]), q = to_f32(w1[k]);
#pragma unroll
            for (int t = 0; t < T; t++) {
                const float xv = job.x[(size_t)t * job.ldx + k];
                a0[t] = fmaf(p, xv, a0[t]);
                a1[t] = fmaf(q, xv, a1[t]);
            }
        }
    }
#pragma unroll
    for (int t = 0; t < T; t++) a0[t] = warp_sum(a0[t]), a1[t] = warp_sum(a1[t]);
    if (ks > 1) {
        if (lane == 0)
#pragma unroll
            for (int t = 0; t < T; t++) s_part[warp][0][t] = a0[t], s_part[warp][1][t] = a1[t];
        __syncthreads();
        if (lane == 0 && part == 0)
            for (int w = 1; w < ks; w++)
#pragma unroll
                for (int t = 0; t < T; t++) a0[t] += s_part[warp + w][0][t], a1[t] += s_part[warp + w][1][t];
    }
    if (lane == 0 && live && part == 0) {
#pragma unroll
        for (int t = 0; t < T; t++) {
            float *y = job.y + (size_t)t * job.ldy + r0;
            if (pair) {
                y[0] = gate_act(job.act, a0[t]) * a1[t];
            } else {
                y[0] = a0[t];
                if (two) y[1] = a1[t];
            }
        }
    }
}

// ---- many tokens, tcgen05 -----------------------------------------------------------------------
// Weights are the M operand (tensor-memory lane = row), tokens the N operand, f32 accumulators.  K advances 64 per stage, in
// the 128-byte swizzle the descriptors expect, zeros past either end.  Every wait is bounded; after a timeout the error flag
// is set, the copies in flight are waited for and the tensor memory is freed.
constexpr int DG_ROWS = 128, DG_K = 64;
constexpr uint32_t DG_W_BYTES = DG_ROWS * 128;

struct DenseGemmJob {
    void *y;             // [seq][ld]
    const float *decay_bias;   // not null: y = decay_of(w x + bias[row])
    float inv_tau;
    int rows, cols, tile0, out_bf16, pair, ld, act, decay_kind;
};
struct DenseGemmJobs {
    DenseGemmJob j[DENSE_MAX_JOBS];
    int n, seq;
};
struct DenseMaps {   // per job: tokens, weights, second weights
    PgTensorMap x[DENSE_MAX_JOBS], w[DENSE_MAX_JOBS], w2[DENSE_MAX_JOBS];
};

// true if all 128 threads of the named barrier bring true
__device__ __forceinline__ bool dq_agree(int barrier, bool v) {
    uint32_t all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.cta.red.and.pred q, %2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(all)
                 : "r"((uint32_t)v), "r"(barrier)
                 : "memory");
    return all != 0;
}
template <class OT>
__device__ __forceinline__ void dg_store(void *y, size_t idx, float v) { reinterpret_cast<OT *>(y)[idx] = from_f32<OT>(v); }

// A pair of CTAs (a cluster of two) multiplies 256 rows x up to 512 tokens: each CTA takes 128 rows (64 of gate and 64 of up
// in the pair form) and half of the tokens, the MMAs read the token halves of both SMs, and a CTA's rows x tokens fill its
// tensor memory (parts of n1 and n2 tokens).  A stage of K moves 48 KB into an SM per 1024 cycles of the tensor pipe; a
// CTA by itself with 256 tokens moved 48 KB per 512 cycles, more than an SM gets from L2.  Four stages.
// Persistent: a pair walks its tiles, token tiles fastest, so that a weight matrix larger than L2 crosses DRAM once.  Warp 0
// issues the copies (the first stages' weights before the dependency wait), warp 1 of the even CTA the MMAs, warps 2-9 read
// the accumulators back, four per part; a part of the next tile starts when its columns are free.
constexpr int DQ_STAGES = 4, DQ_THREADS = 320, DQ_TOK = 512;   // DQ_TOK: most tokens of a tile
constexpr uint32_t DQ_STAGE_BYTES = DQ_TOK / 2 * 128 + DG_W_BYTES;
constexpr uint32_t DQ_EXCHANGE = 2 * 2 * 4 * 8 * 32 * 4;   // parts x buffers in turn x warps x tokens x rows
constexpr size_t DQ_SMEM = (size_t)DQ_STAGES * DQ_STAGE_BYTES + DQ_EXCHANGE + 1024;
struct DenseMapsPair {   // per job: tokens of part 1 and 2 (boxes of n1 / 2 and n2 / 2), weights, second weights
    PgTensorMap x1[DENSE_MAX_JOBS], x2[DENSE_MAX_JOBS], w[DENSE_MAX_JOBS], w2[DENSE_MAX_JOBS];
};
struct DensePair {
    int n1, n2, token_tiles, tiles;   // n1, n2: multiples of 32, at most 256; tiles: pairs of row tiles of all jobs x token tiles
};
RNB_GLOBAL void __launch_bounds__(DQ_THREADS, 1)
dense_gemm_pair_kernel(const __grid_constant__ DenseGemmJobs jobs, const __grid_constant__ DenseMapsPair maps, const DensePair P, int *err_flag) {
    extern __shared__ __align__(1024) uint8_t dg_smem_raw[];
    __shared__ __align__(8) uint64_t full[DQ_STAGES], empty[DQ_STAGES], acc_full, acc_free[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    __shared__ uint32_t s_issued[2];   // of the even CTA: stages that either CTA has asked for
    pdl_launch_dependents();
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(dg_smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)blockIdx.x & 1, pair0 = (int)blockIdx.x >> 1, n_pairs = (int)gridDim.x >> 1, nt = P.n1 + P.n2;
    const uint32_t tok_bytes = (uint32_t)(nt / 2) * 128u, stage_bytes = tok_bytes + DG_W_BYTES;
    if (tid == 0) {
        for (int s = 0; s < DQ_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&acc_full, 1);
        for (int i = 0; i < 2; i++) mbar_init(&acc_free[i], 8);
        mbar_fence_init();
        s_failed = 0;
    }
    if (warp == 1) {
        // no launch that holds tensor memory can share an SM with this much shared memory
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pg_fence_before();
    __syncthreads();
    ps_cluster_sync();   // barriers and tensor memory of both CTAs stand
    pg_fence_after();
    const uint32_t tmem = tmem_slot;
    auto job_of = [&](int tile) {
        int js = 0;
        for (int i = 1; i < jobs.n; i++)
            if (tile / P.token_tiles >= jobs.j[i].tile0) js = i;
        return js;
    };
    // first row of this CTA's part of a tile: rows past the end read as zeros and are never stored
    auto first_row = [&](int tile, const DenseGemmJob &job) { return (2 * (tile / P.token_tiles - job.tile0) + rank) * (job.pair ? DG_ROWS / 2 : DG_ROWS); };
    bool ok = true;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            auto weights = [&](uint32_t at, int js, int kt, int n0) {
                const uint32_t s = at % DQ_STAGES, dst = smem_u32(smem + s * stage_bytes) + tok_bytes, bar = ps_map(smem_u32(&full[s]), 0);
                const bool pair = jobs.j[js].pair != 0;
                if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * stage_bytes);   // both CTAs' copies
                pt_tma_2d(dst, &maps.w[js], kt * DG_K, n0, bar);
                pt_tma_2d(dst + DG_W_BYTES / 2, pair ? &maps.w2[js] : &maps.w[js], kt * DG_K, pair ? n0 : n0 + DG_ROWS / 2, bar);
            };
            int head = 0;
            for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs) {
                const int js = job_of(tile), n0 = first_row(tile, jobs.j[js]), m0 = (tile % P.token_tiles) * nt, KT = (jobs.j[js].cols + DG_K - 1) / DG_K;
                if (tile == pair0) {
                    head = min(KT, DQ_STAGES);
                    for (int kt = 0; kt < head; kt++) weights((uint32_t)kt, js, kt, n0);
                    pdl_wait();   // the tokens are the previous launch's result
                }
                for (int kt = 0; kt < KT; kt++, it++) {
                    const uint32_t s = it % DQ_STAGES, dst = smem_u32(smem + s * stage_bytes), bar = ps_map(smem_u32(&full[s]), 0);
                    if (it >= (uint32_t)head) {
                        ok = mbar_wait_bounded(&empty[s], ((it / DQ_STAGES) & 1u) ^ 1u);
                        if (!ok) break;
                        weights(it, js, kt, n0);
                    }
                    pt_tma_2d(dst, &maps.x1[js], kt * DG_K, m0 + rank * (P.n1 / 2), bar);
                    pt_tma_2d(dst + (uint32_t)(P.n1 / 2) * 128u, &maps.x2[js], kt * DG_K, m0 + P.n1 + rank * (P.n2 / 2), bar);
                }
            }
            ps_st_remote(ps_map(smem_u32(&s_issued[rank]), 0), it);
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t id1 = pt_idesc(P.n1), id2 = pt_idesc(P.n2);
            uint32_t s = 0, phase = 0;
            int count = 0;
            for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs, count++) {
                const int KT = (jobs.j[job_of(tile)].cols + DG_K - 1) / DG_K;
                for (int kt = 0; kt < KT && ok; kt++) {
                    ok = __all_sync(0xffffffffu, pt_wait_shared(&full[s], phase));
                    const uint32_t x1 = smem_u32(smem + s * stage_bytes);
                    const uint64_t dx1 = pg_smem_desc(x1), dx2 = pg_smem_desc(x1 + (uint32_t)(P.n1 / 2) * 128u), dw = pg_smem_desc(x1 + tok_bytes);
                    for (int part = 0; part < 2 && ok; part++) {
                        if (kt == 0 && count > 0) ok = __all_sync(0xffffffffu, pt_wait(&acc_free[part], (uint32_t)((count - 1) & 1)));
                        if (!ok) break;
                        pg_fence_after();
                        if (pg_elect()) {
                            const uint64_t dx = part ? dx2 : dx1;
#pragma unroll
                            for (int k = 0; k < 4; k++) pt_mma(tmem + (uint32_t)part * 256u, dw + 2u * k, dx + 2u * k, part ? id2 : id1, (kt | k) != 0);   // 32 bytes on
                            if (part) pt_commit(&empty[s]);
                        }
                        __syncwarp();
                    }
                    if (++s == DQ_STAGES) s = 0, phase ^= 1u;
                }
                if (ok && pg_elect()) pt_commit(&acc_full);
                __syncwarp();
            }
        }
    } else {
        const int q = warp & 3, part = (warp - 2) >> 2, cols = part ? P.n2 : P.n1;   // tensor-memory lane quarter and columns of this warp
        float *const ex = reinterpret_cast<float *>(smem + (size_t)DQ_STAGES * DQ_STAGE_BYTES + (size_t)part * (DQ_EXCHANGE / 2));
        const uint32_t at = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * 256);
        pdl_wait();   // stores come after the launches before this one
        int turn = 0;
        auto landed = [&](int count) { return __all_sync(0xffffffffu, mbar_wait_bounded(&acc_full, (uint32_t)(count & 1))) != 0; };
        ok = walk_tiles(pair0, n_pairs, P.tiles, landed, [&](bool v) { return dq_agree(1 + part, v); }, [&](int tile) {
            const DenseGemmJob &job = jobs.j[job_of(tile)];
            const int n0 = first_row(tile, job), m0 = (tile % P.token_tiles) * nt + part * P.n1, rows = job.rows;
            pg_fence_after();
            if (job.pair)
                for (int c = 0; c < cols && m0 + c < jobs.seq; c += 16, turn ^= 1) {
                    // gate rows on lanes 0-63, the same rows of up on lanes 64-127: a warp hands eight of 16 tokens to its partner
                    uint32_t v[16];
                    ps_tmem_ld<16>(at + (uint32_t)c, v);
                    const bool up = q >= 2;
                    float *buf = ex + turn * (4 * 8 * 32);
#pragma unroll
                    for (int i = 0; i < 8; i++) buf[((q ^ 2) * 8 + i) * 32 + lane] = __uint_as_float(up ? v[i] : v[8 + i]);
                    asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
                    const int row = n0 + (q & 1) * 32 + lane;
                    if (row < rows) {
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const int tok = m0 + c + i + (up ? 8 : 0);
                            const float other = buf[(q * 8 + i) * 32 + lane], own = __uint_as_float(up ? v[8 + i] : v[i]);
                            const float z = up ? other : own, u = up ? own : other;
                            if (tok >= jobs.seq) continue;
                            const float a = (job.out_bf16 ? gate_act_fast(job.act, z) : gate_act(job.act, z)) * u;
                            if (job.out_bf16) dg_store<bf16>(job.y, (size_t)tok * job.ld + row, a);
                            else dg_store<float>(job.y, (size_t)tok * job.ld + row, a);
                        }
                    }
                }
            else {
                const int row = n0 + q * 32 + lane;
                const float b = job.decay_bias && row < rows ? job.decay_bias[row] : 0.f;
                for (int c = 0; c < cols && m0 + c < jobs.seq; c += 32) {
                    uint32_t v[32];
                    pg_tmem_ld32(at + (uint32_t)c, v);
                    if (row >= rows) continue;
                    if (job.decay_bias) {
                        if (job.decay_kind == DECAY_SIGMOID_ROOT) {
#pragma unroll
                            for (int i = 0; i < 32; i++) v[i] = __float_as_uint(sigmoid_root_fast(__uint_as_float(v[i]) + b, job.inv_tau));
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; i++) v[i] = __float_as_uint(expf(-expf(__uint_as_float(v[i]) + b)));
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        const int tok = m0 + c + i;
                        if (tok < jobs.seq) {
                            if (job.out_bf16) dg_store<bf16>(job.y, (size_t)tok * job.ld + row, __uint_as_float(v[i]));
                            else dg_store<float>(job.y, (size_t)tok * job.ld + row, __uint_as_float(v[i]));
                        }
                    }
                }
            }
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pt_arrive(ps_map(smem_u32(&acc_free[part]), 0));
        });
    }
    if (!ok) s_failed = 1;
    __syncwarp();
    pg_fence_before();
    __syncthreads();
    ps_cluster_sync();   // the other CTA's memory and barriers are no longer used
    if (s_failed) {
        // A CTA that has read its last accumulators knows that all copies have landed.  One that gave up does not: both CTAs' copies count
        // on the even CTA's barriers, and what the odd one asked for beyond the even one's last stage is announced here.  The
        // odd CTA stays for it if it has given up too.
        if (rank == 0 && tid == 0) {
            for (uint32_t i = s_issued[0]; i < s_issued[1]; i++) mbar_arrive_expect_tx(&full[i % DQ_STAGES], stage_bytes);
            pg_drain(full, max(s_issued[0], s_issued[1]), DQ_STAGES);
        }
        __syncthreads();
        ps_cluster_sync();
    }
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
        if (lane == 0 && s_failed && err_flag) atomicExch(err_flag, DEV_ERR_GEMM_TIMEOUT);
    }
}

// ---- some tokens, tcgen05, K cut over a cluster --------------------------------------------------
// A tile of 128 rows x nt tokens (a multiple of 16, at most 256) belongs to the ks CTAs of a cluster; each multiplies its
// part of K and they add their accumulators over distributed shared memory in rank order (ps_reduce).  Fewer tokens leave
// room for more stages, so that the weights stream.  The first stages' weights are asked for before the dependency wait.
// What bounds it: the stream of the weights, and the fill and drain of a launch.  An output and down projection of 2048
// rows gave the 256-token tiles 16 CTAs at 150 tokens; a prompt of 64 tokens through 8 Punisun layers of width 2048 takes
// 1.46 ms (2.45 with those tiles), one of 150 through 6 Dutivik layers 1.06 ms (1.58).
// Warp 0 issues the copies, warp 1 the MMAs, warps 2-5 reduce and store.  grid = (row tiles of all jobs x ks, token tiles).
constexpr int DP_SUB = 16, DP_MAX_STAGES = 5, DP_THREADS = 192, DP_TOK = 256;   // DP_TOK: most tokens per CTA
constexpr size_t DP_SMEM = PS_SMEM;   // two CTAs per SM
struct DenseSplit {
    int nt, stages, ks;
    uint32_t tmem_cols;
};
RNB_GLOBAL void __launch_bounds__(DP_THREADS)
dense_gemm_split_kernel(const __grid_constant__ DenseGemmJobs jobs, const __grid_constant__ DenseMaps maps, const DenseSplit P, int *err_flag) {
    extern __shared__ __align__(1024) uint8_t dg_smem_raw[];
    __shared__ __align__(8) uint64_t full[DP_MAX_STAGES], empty[DP_MAX_STAGES], done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    pdl_launch_dependents();
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(dg_smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = (int)blockIdx.x / P.ks, kr = (int)blockIdx.x - tile * P.ks;
    int js = 0;
    for (int i = 1; i < jobs.n; i++)
        if (tile >= jobs.j[i].tile0) js = i;
    const DenseGemmJob &job = jobs.j[js];
    const bool pair = job.pair != 0;
    const int rows = job.rows, S = P.stages;
    const int n0 = (tile - job.tile0) * (pair ? DG_ROWS / 2 : DG_ROWS), m0 = blockIdx.y * P.nt, end = min(jobs.seq, m0 + P.nt);
    const int all = (job.cols + DG_K - 1) / DG_K, k0 = all * kr / P.ks, KT = all * (kr + 1) / P.ks - k0;   // this CTA's stages of K
    const uint32_t x_bytes = (uint32_t)P.nt * 128u, stage_bytes = x_bytes + DG_W_BYTES;
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&done_bar, 1);
        mbar_fence_init();
        s_failed = 0;
    }
    __syncthreads();
    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            auto weights = [&](int kt) {
                const uint32_t dst = smem_u32(smem + (uint32_t)(kt % S) * stage_bytes) + x_bytes;
                uint64_t *bar = &full[kt % S];
                mbar_arrive_expect_tx(bar, stage_bytes);
                pg_tma_2d(dst, &maps.w[js], (k0 + kt) * DG_K, n0, bar);
                pg_tma_2d(dst + DG_W_BYTES / 2, pair ? &maps.w2[js] : &maps.w[js], (k0 + kt) * DG_K, pair ? n0 : n0 + DG_ROWS / 2, bar);
            };
            const int head = min(S, KT);
            for (int kt = 0; kt < head; kt++) weights(kt);
            pdl_wait();   // the tokens are the previous launch's result
            int issued = 0;
            for (int kt = 0; kt < KT && ok; kt++) {
                const int s = kt % S;
                if (kt >= S) {
                    ok = mbar_wait_bounded(&empty[s], (uint32_t)(((kt / S) & 1) ^ 1));
                    if (!ok) break;
                    weights(kt);
                }
                pg_tma_2d(smem_u32(smem + (uint32_t)s * stage_bytes), &maps.x[js], (k0 + kt) * DG_K, m0, &full[s]);
                issued = kt + 1;
            }
            pg_drain(full, (uint32_t)issued, (uint32_t)S);   // the stages are reused
        }
    } else if (warp == 1) {
        pdl_wait();   // tensor memory is asked for when no earlier launch can still hold it
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(P.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        __syncwarp();
        const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(&tmem_slot);
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(P.nt >> 3) << 17) | ((uint32_t)(DG_ROWS >> 4) << 24);
        for (int kt = 0; kt < KT && ok; kt++) {
            const int s = kt % S;
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&full[s], (uint32_t)((kt / S) & 1)));
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
        }
        if (ok && pg_elect()) pg_commit(&done_bar);
        __syncwarp();
    }
    if (!ok) s_failed = 1;
    __syncthreads();   // the accumulators' address; a failure of any role
    pdl_wait();        // every thread that stores comes after the launches before this one
    const bool fin = __all_sync(0xffffffffu, s_failed == 0 && mbar_wait_bounded(&done_bar, 0u));
    if (!fin) s_failed = 1;
    pg_fence_after();
    const uint32_t tmem = tmem_slot;
    if (P.ks > 1) ps_cluster_sync();   // every CTA's MMAs have read their stages: the slots may be written
    const int q = warp & 3;
    float *ex = reinterpret_cast<float *>(smem + PS_SLOT_BYTES);   // gate / up exchange, two buffers in turn
    ps_reduce<DP_SUB, 1>(P.ks, kr, (end - m0 + DP_SUB - 1) / DP_SUB, smem, tmem, warp >= 2, q, 0, fin, [&](int cc, int j, const float (&v)[DP_SUB]) {
        const int tok0 = m0 + cc * DP_SUB;
        auto put = [&](int t, int row, float a) {
            if (tok0 + t >= end) return;
            if (job.out_bf16) dg_store<bf16>(job.y, (size_t)(tok0 + t) * job.ld + row, a);
            else dg_store<float>(job.y, (size_t)(tok0 + t) * job.ld + row, a);
        };
        if (pair) {
            // gate rows on lane quarters 0 and 1, the same rows of up on 2 and 3: each warp finishes half of the tokens
            float *buf = ex + (size_t)(j & 1) * (DP_SUB * DG_ROWS);
#pragma unroll
            for (int t = 0; t < DP_SUB; t++) buf[t * DG_ROWS + q * 32 + lane] = v[t];
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const int row = n0 + (q & 1) * 32 + lane, t_lo = (q >> 1) * (DP_SUB / 2);
            if (fin && row < rows) {
#pragma unroll
                for (int t = t_lo; t < t_lo + DP_SUB / 2; t++) {
                    const float z = buf[t * DG_ROWS + (q & 1) * 32 + lane], u = buf[t * DG_ROWS + 64 + (q & 1) * 32 + lane];
                    put(t, row, (job.out_bf16 ? gate_act_fast(job.act, z) : gate_act(job.act, z)) * u);
                }
            }
        } else if (fin && n0 + q * 32 + lane < rows) {
            const int row = n0 + q * 32 + lane;
            const float b = job.decay_bias ? job.decay_bias[row] : 0.f;
#pragma unroll
            for (int t = 0; t < DP_SUB; t++)
                put(t, row, !job.decay_bias ? v[t] : job.decay_kind == DECAY_SIGMOID_ROOT ? sigmoid_root_fast(v[t] + b, job.inv_tau) : expf(-expf(v[t] + b)));
        }
    });
    pg_fence_before();
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P.tmem_cols) : "memory");
        if (lane == 0 && s_failed && err_flag) atomicExch(err_flag, DEV_ERR_GEMM_TIMEOUT);
    }
}

// ---- many tokens, f32 arithmetic on the CUDA cores ----------------------------------------------
struct DenseSimtJob {
    const bf16 *w, *w2;
    const void *x;       // [seq][ldx] of XT
    void *y;             // [seq][ld]
    int rows, cols, tile0, out_bf16, ldx, ld, act;
};
struct DenseSimtJobs {
    DenseSimtJob j[DENSE_MAX_JOBS];
    int n, seq;
};
constexpr int DS_TILE = 64, DS_K = 16;
// grid = (row tiles of all jobs, token tiles), 256 threads, a 4 x 4 block of outputs per thread
template <class XT>
RNB_GLOBAL void __launch_bounds__(256)
dense_gemm_simt_kernel(const __grid_constant__ DenseSimtJobs jobs) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float xs[DS_K][DS_TILE + 4], ws[DS_K][DS_TILE + 4], us[DS_K][DS_TILE + 4];
    int js = 0;
    for (int i = 1; i < jobs.n; i++)
        if ((int)blockIdx.x >= jobs.j[i].tile0) js = i;
    const DenseSimtJob &job = jobs.j[js];
    const bool pair = job.w2 != nullptr;
    const XT *x = reinterpret_cast<const XT *>(job.x);
    const int n0 = ((int)blockIdx.x - job.tile0) * DS_TILE, m0 = blockIdx.y * DS_TILE;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    float a[4][4] = {}, b[4][4] = {};
    for (int k0 = 0; k0 < job.cols; k0 += DS_K) {
        for (int i = tid; i < DS_TILE * DS_K; i += 256) {
            const int k = i & (DS_K - 1), r = i / DS_K;
            const bool kin = k0 + k < job.cols;
            xs[k][r] = kin && m0 + r < jobs.seq ? to_f32(x[(size_t)(m0 + r) * job.ldx + k0 + k]) : 0.f;
            const bool win = kin && n0 + r < job.rows;
            ws[k][r] = win ? to_f32(job.w[(size_t)(n0 + r) * job.cols + k0 + k]) : 0.f;
            if (pair) us[k][r] = win ? to_f32(job.w2[(size_t)(n0 + r) * job.cols + k0 + k]) : 0.f;
        }
        __syncthreads();
        float c[4][4] = {}, d[4][4] = {};   // sums of sums: rounding grows with the depth of one tile and the number of tiles
#pragma unroll
        for (int k = 0; k < DS_K; k++) {
            const float4 xv = *reinterpret_cast<const float4 *>(&xs[k][ty * 4]), wv = *reinterpret_cast<const float4 *>(&ws[k][tx * 4]);
            const float xr[4] = {xv.x, xv.y, xv.z, xv.w}, wr[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) c[i][j] = fmaf(xr[i], wr[j], c[i][j]);
            if (pair) {
                const float4 uv = *reinterpret_cast<const float4 *>(&us[k][tx * 4]);
                const float ur[4] = {uv.x, uv.y, uv.z, uv.w};
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) d[i][j] = fmaf(xr[i], ur[j], d[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) a[i][j] += c[i][j], b[i][j] += d[i][j];
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int tok = m0 + ty * 4 + i, row = n0 + tx * 4 + j;
            if (tok >= jobs.seq || row >= job.rows) continue;
            const float v = pair ? gate_act(job.act, a[i][j]) * b[i][j] : a[i][j];
            if (job.out_bf16) dg_store<bf16>(job.y, (size_t)tok * job.ld + row, v);
            else dg_store<float>(job.y, (size_t)tok * job.ld + row, v);
        }
}

}  // namespace rnb
