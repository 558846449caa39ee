// Prefill matmul on pairs of SMs (tcgen05, cta_group::2): dequantised bf16 weights from tensor memory x bf16 tokens from
// shared memory, f32 accumulators.
//
// A pair of CTAs multiplies 256 weight rows x up to 256 tokens: each CTA dequantises its own 128 rows, brings in half of the
// tokens, and holds its rows' accumulators in the first 256 columns of its tensor memory.  The other 256 columns are a ring of
// weights, two blocks of K deep (64 elements = 32 columns): a thread dequantises the 64 elements of a row in registers and
// writes them to the row's lane.  Tiles of up to 384 tokens (two MMAs, a ring of one block) dequantise less where the chip stays
// full.  Weights as an operand in shared memory have every stage behind a proxy fence and, in the odd CTA, behind a release across the
// cluster (prefill_gemm_wide.cuh); tensor memory needs neither (tcgen05.wait::st, a tcgen05 fence and a relaxed arrival at the even
// CTA's barrier), and what the dequantising warps cost is their instructions.
//
// Blocks of 256 elements of the 128 rows come into shared memory as they are, by tiled copies, up to three ahead; a group of
// four warps (128 rows) takes one of a block's four stages.  Both CTAs' token copies count on the even CTA's barriers.  One
// commit frees a stage of tokens and of weights in both CTAs.
//
// ks = 1: persistent, a pair walks its tiles (token tiles fastest, so that a weight row crosses DRAM once); behind the first
// block of the next tile the dequantising warps read the finished one from tensor memory, hand the columns back, and store.
// ks > 1: K is cut over the ks pairs of a cluster, one tile each; they add their accumulators over distributed shared memory
// in rank order (the same bits on every run).
//
// Warps 0-15 dequantise and store, warp 16 of the even CTA issues the MMAs, warp 17 of each CTA the token copies, warp 18 those
// of the weights.  The MMAs wait for half a block at a time: with a wait a stage their loop takes 2900 cycles a block, more than the rest.
// Every wait is bounded; after a timeout all threads still meet at the cluster barrier.
//
// What bounds it: the issue slots of the dequantising warps (Q4_K 407 to 424 warp instructions a block and warp, the way back of the
// tile included; a block takes 1.1 us, 1.23 with every SM at work, of Q6_K 1.45 and 1.6), from about 200 tokens a tile on the tensor pipe.
// Measured with 203 / 511 / 2048 tokens, us, cold, with the conversion of the tokens to bf16 (weights in shared memory before): gate + up
// 28672 x 4096 60 / 110 / 335 (89 / 114 / 372), down 4096 x 14336 Q6_K 50 / 71 / 190 (68 / 116 / 191), q + k + v 32 / 44 / 89 (48 / 54 / 103), o
// 26 / 32 / 69 (40 / 48 / 69).  ncu, 2048 tokens: gate + up 354 us = 1357 TFLOP/s = 0.82 of the measured 1658, tensor pipe 80 % and issue
// slots 67 % of the active cycles; o 65 and 56 %, q + k + v 70 and 46 %.
#pragma once
#include "prefill_gemm.cuh"
#include "prefill_gemm_split.cuh"

namespace rnb {

constexpr int PT_STAGES = 4;       // half blocks of K: two blocks; one above 256 tokens
constexpr int PT_WORKERS = 16;     // dequantising warps
constexpr int PT_THREADS = (PT_WORKERS + 3) * 32;
constexpr int PT_TOK = 384;        // most tokens of a tile, 256 of one with the deeper ring
constexpr int PT_MAX_KS = 4;       // pairs per cluster
// Blocks of 128 rows as they are in memory: Q4_K 144 bytes a row; Q6_K 240, from the last 16-byte boundary before its 210 bytes
constexpr int PT_RAWS = 3;
constexpr uint32_t PT_Q4_PITCH = Q4K_BYTES, PT_Q6_PITCH = 240, PT_RAW_BYTES = PG_ROWS * PT_Q6_PITCH;
constexpr uint32_t PT_RING = PT_STAGES * 2 * (256 / 2 * 128);   // tokens; the reduction over a cluster reuses it
static_assert(PT_STAGES / 2 * 2 * (PT_TOK / 2 * 128) <= PT_RING, "tokens of the widest tile");
constexpr size_t PT_SMEM = PT_RING + PT_RAWS * PT_RAW_BYTES + 1024;

struct PtParams {
    int seq, cols, nt, ks;             // nt: tokens of a tile (a multiple of 16 up to 256, of 32 up to PT_TOK), ks: pairs along K
    int row_tiles, token_tiles, tiles; // tiles: pairs of row tiles x token tiles
    int skew;                          // bit i: job i's rows start at any even address (Q6_K)
};
// Tokens (boxes of half a part of a tile: up to 256 tokens are one part, more are two); blocks of each job's rows, and of the second
// matrix of a pair: boxes of 64 rows.  Skewed rows have a map for every eighth row (they lie a multiple of 16 bytes apart), from the 16-byte
// boundary before its first byte: boxes of 16, 8 in a pair.
struct PtMaps {
    PgTensorMap x, w[PG_MAX_JOBS][8], w2[8];
};

// An arrival at another CTA's barrier, and a wait for one: they order what either CTA did before it.
__device__ __forceinline__ void pt_arrive(uint32_t cluster_addr) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory"); }
// The same for what lies in shared memory alone, and behind tcgen05.wait and tcgen05.fence::before_thread_sync in tensor memory.  As
// a thread's release of all its memory an arrival takes over 1000 cycles.
__device__ __forceinline__ void pt_arrive_shared(uint32_t cluster_addr) {
    asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n\tmbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
template <bool SHARED>
__device__ __forceinline__ bool pt_wait_in(uint64_t *bar, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 22); i++) {
        uint32_t done;
        if constexpr (SHARED)
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(done)
                         : "r"(smem_u32(bar)), "r"(parity)
                         : "memory");
        else
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(done)
                         : "r"(smem_u32(bar)), "r"(parity)
                         : "memory");
        if (done) {
            if constexpr (SHARED) asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
            return true;
        }
        if (i > 64) __nanosleep(i > 4096 ? 256 : 32);
    }
    return false;
}
__device__ __forceinline__ bool pt_wait(uint64_t *bar, uint32_t parity) { return pt_wait_in<false>(bar, parity); }
__device__ __forceinline__ bool pt_wait_shared(uint64_t *bar, uint32_t parity) { return pt_wait_in<true>(bar, parity); }
// Both of two barriers of the pair, asked at the same time: a wait takes some 200 cycles even when there is nothing to wait for.
__device__ __forceinline__ bool pt_wait_shared(uint64_t *a, uint64_t *b, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 22); i++) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p, q;\n\tmbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %3;\n\t"
                     "mbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 q, [%2], %3;\n\tand.pred p, p, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(smem_u32(a)), "r"(smem_u32(b)), "r"(parity)
                     : "memory");
        if (done) {
            asm volatile("fence.acquire.sync_restrict::shared::cluster.cluster;" ::: "memory");
            return true;
        }
        if (i > 64) __nanosleep(i > 4096 ? 256 : 32);
    }
    return false;
}
// A warp's wait, with one outcome for all lanes
__device__ __forceinline__ bool pt_warp_wait(uint64_t *bar, uint32_t parity) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity));
}
// D += A x B; A in shared memory, in tensor memory
__device__ __forceinline__ void pt_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void pt_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void pt_tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
        "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
        "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
// the barrier at the same place in both CTAs of the pair whose even CTA has rank `even` in the cluster
__device__ __forceinline__ void pt_commit(uint64_t *bar, int even = 0) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)(3 << even)) : "memory");
}
// tiled copy into this CTA that counts on a barrier of either CTA of the pair
__device__ __forceinline__ void pt_tma_2d(uint32_t dst, const void *tmap, int x, int y, uint32_t cluster_bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(cluster_bar)
                 : "memory");
}
// instruction descriptor: D = f32, A = B = bf16, both K-major, M = 256 (128 rows of each CTA), N = n
__device__ __forceinline__ uint32_t pt_idesc(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24); }

// ---- a stage's 64 elements of a row, from the block in shared memory into registers ---------------
// o[j] = elements 2j and 2j + 1 of stage g; the arithmetic of pg_dequant_q4 and pg_dequant_q6_half.  read(): the block's bytes
// have been read.
// a * b + c, a and b in f16, rounded once to f32
__device__ __forceinline__ float pt_fma_f16(__half a, __half b, float c) {
    float r;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(r) : "h"(__half_as_ushort(a)), "h"(__half_as_ushort(b)), "f"(c));
    return r;
}
// Bits of two bytes 16 bits apart, as f16 of 1024 + (byte & mask).  One instruction: from C the mask and the
// exponent become two.
__device__ __forceinline__ __half2 pt_nibbles(uint32_t word, uint32_t mask) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(word), "r"(mask), "r"(0x64006400u));   // (word & mask) | exponent
    return *reinterpret_cast<const __half2 *>(&r);
}
template <class F>
__device__ __forceinline__ void pt_dequant_q4(const uint8_t *blk, int g, uint32_t (&o)[32], F &&read) {
    const uint4 hdr = *reinterpret_cast<const uint4 *>(blk), q0 = *reinterpret_cast<const uint4 *>(blk + 16 + 32 * g), q1 = *reinterpret_cast<const uint4 *>(blk + 32 + 32 * g);
    read();
    const float dmin = f16_bits_to_f32(hdr.x >> 16);
    const uint32_t scw = g < 2 ? hdr.y & 0x3f3f3f3fu : (hdr.w & 0x0f0f0f0fu) | (((hdr.y >> 6) & 0x03030303u) << 4);
    const uint32_t mnw = g < 2 ? hdr.z & 0x3f3f3f3fu : ((hdr.w >> 4) & 0x0f0f0f0fu) | (((hdr.z >> 6) & 0x03030303u) << 4);
    const uint32_t ql[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    const __half dh = __ushort_as_half((unsigned short)(hdr.x & 0xffffu));
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int sh = 16 * (g & 1) + 8 * h;
        const float nm = -__fmul_rn(dmin, (float)((mnw >> sh) & 0xffu));
        // nibble x scale in f16, at most 945 and so exact: (1024 + q) sc - 1024 sc, of a high nibble (1024 + 16 q) sc / 16 - 64 sc
        const __half sc = __ushort2half_rn((unsigned short)((scw >> sh) & 0xffu));
        const __half2 s2 = __half2half2(h ? __hmul(sc, __float2half(0.0625f)) : sc), c2 = __half2half2(__hmul(sc, __float2half(h ? -64.f : -1024.f)));
        const uint32_t mask = h ? 0x00f000f0u : 0x000f000fu;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const __half2 e = __hfma2(pt_nibbles(ql[w], mask), s2, c2), f = __hfma2(pt_nibbles(ql[w] >> 8, mask), s2, c2);   // bytes 0 and 2, 1 and 3
            o[16 * h + 2 * w] = pg_pack_bf16(pt_fma_f16(__low2half(e), dh, nm), pt_fma_f16(__low2half(f), dh, nm));
            o[16 * h + 2 * w + 1] = pg_pack_bf16(pt_fma_f16(__high2half(e), dh, nm), pt_fma_f16(__high2half(f), dh, nm));
        }
    }
}
// Q6_K at any even address: bytes by aligned 16-byte windows, shifted into place.
template <class F>
__device__ __forceinline__ void pt_dequant_q6(const uint8_t *blk, int g, uint32_t (&o)[32], F &&read) {
    const int n = g >> 1, ls = 4 * (g & 1);
    uint32_t qh[8];
    pg_ldg_window<8, 3, true>(blk + 128 + 32 * n, qh);
    const uint16_t *sc = reinterpret_cast<const uint16_t *>(blk + 192 + 4 * g);
    const uint32_t s2[2] = {sc[0], sc[1]};
    const float d = f16_bits_to_f32(*reinterpret_cast<const uint16_t *>(blk + 208));
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t ql[8];
        pg_ldg_window<8, 3, true>(blk + 64 * n + 32 * h, ql);
        if (h == 1) read();
        const float ds0 = __fmul_rn(d, (float)(int)(int8_t)(s2[h] & 0xffu)), ds1 = __fmul_rn(d, (float)(int)(int8_t)(s2[h] >> 8));
        const uint64_t sp[2] = {pg_pair_f32(ds0, ds0), pg_pair_f32(ds1, ds1)};
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const uint32_t n6 = ((ql[w] >> ls) & 0x0f0f0f0fu) | (((qh[w] >> (ls + 2 * h)) << 4) & 0x30303030u);
            o[16 * h + 2 * w] = pg_dequant_pair_mul_m32(n6, 0, sp[w >> 2]);
            o[16 * h + 2 * w + 1] = pg_dequant_pair_mul_m32(n6, 2, sp[w >> 2]);
        }
    }
}
// The same where all rows of a warp have their block at 4 K + 2 odd bytes behind a 16-byte boundary (base): which words are needed
// is known.  An element's six bits in a byte become f16 of 1024 + q by one permutation for two; d times that less what is too
// much, and its product with the scale, are exact in f32, as they are above.  d is finite: else that difference is NaN for every q.
template <int K, class F>
__device__ __forceinline__ void pt_dequant_q6_at(const uint8_t *base, uint32_t odd, int g, uint32_t (&o)[32], F &&read) {
    const int n = g >> 1;
    const uint32_t sh = 16u * odd + 4u * (g & 1);   // to a word's bytes, and in odd groups to their high nibbles
    auto window = [&](uint32_t at, uint32_t (&v)[12]) {
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const uint4 t = *reinterpret_cast<const uint4 *>(base + at + 16 * j);
            v[4 * j] = t.x, v[4 * j + 1] = t.y, v[4 * j + 2] = t.z, v[4 * j + 3] = t.w;
        }
    };
    uint32_t v[12], qh[8];
    window(128 + 32 * n, v);
#pragma unroll
    for (int w = 0; w < 8; w++) qh[w] = __funnelshift_r(v[w + K], v[w + K + 1], sh);   // bits 0-1 of a byte: of the first half, 2-3: of the second
    const uint8_t *blk = base + 4 * K + 2 * odd;
    const uint16_t *sc = reinterpret_cast<const uint16_t *>(blk + 192 + 4 * g);
    const uint32_t s2[2] = {sc[0], sc[1]};
    const __half d = __ushort_as_half(*reinterpret_cast<const unsigned short *>(blk + 208));
    const float off = __fmul_rn(__half2float(d), -1056.f);
#pragma unroll
    for (int h = 0; h < 2; h++) {
        window(64 * n + 32 * h, v);
        if (h == 1) read();
        const float sc0 = (float)(int)(int8_t)(s2[h] & 0xffu), sc1 = (float)(int)(int8_t)(s2[h] >> 8);
        const uint64_t sp[2] = {pg_pair_f32(sc0, sc0), pg_pair_f32(sc1, sc1)};
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const uint32_t lo = __funnelshift_r(v[w + K], v[w + K + 1], sh);
            uint32_t q = h ? qh[w] << 2 : qh[w] << 4;
            asm("lop3.b32 %0, %0, 0x30303030, 0, 0xc0;" : "+r"(q));
            asm("lop3.b32 %0, %1, 0x0f0f0f0f, %0, 0xea;" : "+r"(q) : "r"(lo));   // (lo & mask) | q
            auto pair = [&](uint32_t e) {
                const __half2 f = *reinterpret_cast<const __half2 *>(&e);
                uint32_t r;
                asm("{\n\t.reg .b64 t;\n\t.reg .b32 x, y;\n\tmov.b64 t, {%1, %2};\n\tmul.rn.f32x2 t, t, %3;\n\tmov.b64 {x, y}, t;\n\tcvt.rn.bf16x2.f32 %0, y, x;\n\t}"
                    : "=r"(r)
                    : "f"(pt_fma_f16(__low2half(f), d, off)), "f"(pt_fma_f16(__high2half(f), d, off)), "l"(sp[w >> 2]));
                return r;
            };
            o[16 * h + 2 * w] = pair(__byte_perm(q, 0x64646464u, 0x4140));
            o[16 * h + 2 * w + 1] = pair(__byte_perm(q, 0x64646464u, 0x4342));
        }
    }
}
// Row of a tile (of each matrix of a pair: lanes 0-15 the first, the others the second) that a lane of quarter q holds, and where the
// row's block stands.  Skewed rows come from eight copies: the lanes of a bank phase take rows of different places in a copy.
__device__ __forceinline__ int pt_row(bool pair, bool skew, int q) {
    const int lane = threadIdx.x & 31;
    if (!skew) return pair ? q * 16 + (lane & 15) : q * 32 + lane;
    return pair ? q * 16 + 8 * (lane & 1) + ((lane >> 1) & 7) : q * 32 + 8 * (lane & 3) + (lane >> 2);
}
__device__ __forceinline__ int pt_place(bool pair, bool skew, int row) {
    return (skew ? (row & 7) * (pair ? 8 : 16) + (row >> 3) : row) + (pair && (threadIdx.x & 16) ? PG_ROWS / 2 : 0);
}

// Some tokens of a row from registers.  Gate + up: lanes 0-15 hold gate rows, 16-31 the same rows of up; the two lanes of a row
// finish a token each.
template <int N>
__device__ __forceinline__ void pt_store(const PgJob &job, int r, int tok0, int seq, const uint32_t (&v)[N]) {
    const int lane = threadIdx.x & 31, rows = job.rows;
    if (job.w2) {
        const int up = lane >> 4;
        uint16_t *dst = job.yb + (size_t)(tok0 + up) * rows + r;
#pragma unroll
        for (int j = 0; j < N; j += 2) {
            const float own = __uint_as_float(up ? v[j + 1] : v[j]);
            const float other = __uint_as_float(__shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + 1], 16));
            const float g = up ? other : own, u = up ? own : other;
            // fast exponential and division: their 2^-21 relative error disappears in the bf16 rounding below
            const float a = __fdividef(g, 1.0f + __expf(-g)) * u;
            if (r < rows && tok0 + up + j < seq) *dst = (uint16_t)(pg_pack_bf16(a, 0.f) & 0xffffu);
            dst += 2 * (size_t)rows;
        }
    } else {
        float *dst = job.y + (size_t)tok0 * rows + r;
        if (r < rows) {
#pragma unroll
            for (int j = 0; j < N; j++) {
                if (tok0 + j < seq) *dst = __uint_as_float(v[j]);
                dst += rows;
            }
        }
    }
}

// CUT: ks > 1, a cluster per tile.  grid = 2 x ks x pairs, cluster (2 ks, 1, 1).  PT_THREADS threads; dynamic shared memory PT_SMEM.
template <bool CUT>
RNB_GLOBAL void __launch_bounds__(PT_THREADS, 1)
prefill_gemm_pair_kernel(const __grid_constant__ PgJobs jobs, const __grid_constant__ PtMaps maps, const PtParams P, int *err_flag) {
    extern __shared__ __align__(1024) uint8_t pg_smem_raw[];
    // weights written (both CTAs' warps), tokens landed (both CTAs' copies), stage free; blocks landed, read; accumulators complete, read
    __shared__ __align__(8) uint64_t w_full[PT_STAGES], full[PT_STAGES], empty[PT_STAGES], raw_full[PT_RAWS], raw_empty[PT_RAWS], acc_full, acc_free;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_failed;
    __shared__ uint32_t s_issued[2];   // of the even CTA: token stages that either CTA has asked for
    pdl_launch_dependents();
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(pg_smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int ks = CUT ? P.ks : 1, rank = (int)blockIdx.x & 1, kr = CUT ? ((int)blockIdx.x >> 1) % ks : 0, even = 2 * kr, pair0 = (int)blockIdx.x / (2 * ks),
              n_pairs = (int)gridDim.x / (2 * ks);
    const int nb_row = P.cols >> 8, b0 = nb_row * kr / ks, nb = nb_row * (kr + 1) / ks - b0;   // this pair's blocks of K
    const int parts = P.nt > 256 ? 2 : 1, part = P.nt / parts;   // tokens of an MMA; a CTA brings in half of them
    const uint32_t half_bytes = (uint32_t)(part / 2) * 128u, panel = (uint32_t)parts * half_bytes, stage_bytes = 2 * panel;   // 64, 64, 128 elements of K
    const uint32_t ring = parts == 2 ? PT_STAGES / 2 : PT_STAGES, ring_log = parts == 2 ? 1 : 2, w_col = parts == 2 ? PT_TOK : 256;   // weights behind the accumulators
    if (tid == 0) {
        for (int s = 0; s < PT_STAGES; s++) {
            mbar_init(&w_full[s], 16);   // two groups of four warps of each CTA
            mbar_init(&full[s], 1);   // the even CTA's announcement of both CTAs' bytes
            mbar_init(&empty[s], 1);    // tcgen05.commit
        }
        for (int s = 0; s < PT_RAWS; s++) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], PT_WORKERS);
        }
        mbar_init(&acc_full, 1);
        mbar_init(&acc_free, 2 * PT_WORKERS);
        mbar_fence_init();
        s_failed = 0;
    }
    if (warp == PT_WORKERS) {
        // no launch that holds tensor memory can share an SM with this much shared memory
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pg_fence_before();
    __syncthreads();
    ps_cluster_sync();   // barriers and tensor memory of all CTAs stand
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
    // row of its matrix that a lane of a dequantising warp holds
    auto row_of = [&](int tile) {
        int local;
        const int js = job_of(tile, local);
        const bool pair = jobs.j[js].w2 != nullptr;
        return local * (pair ? PG_ROWS / 2 : PG_ROWS) + pt_row(pair, (P.skew >> js) & 1, warp & 3);
    };
    // an odd number of row tiles: the last odd CTA multiplies a tile twice and does not store
    auto mine = [&](int tile) { return 2 * (tile / P.token_tiles) + rank < P.row_tiles; };
    const int grp = (warp >> 2) & 3, q = warp & 3;   // of a dequantising warp: stage of a block, quarter of the tensor-memory lanes
    bool ok = true;

    if (warp < PT_WORKERS) {
        uint32_t uses = 0, rs = 0, rphase = 0;   // blocks so far; slot of the ring of raw blocks
        const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
        // tile `tile`, the pair's `count`-th: a warp takes every fourth group of 32 tokens
        auto finish = [&](int tile, int count) {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&acc_full, (uint32_t)(count & 1)));
            if (!ok) return;
            pg_fence_after();
            const int row = row_of(tile), m0 = (tile % P.token_tiles) * P.nt, end = min(P.seq, m0 + P.nt);
            int local;
            const PgJob &job = jobs.j[job_of(tile, local)];
            uint32_t v[2][32];
            auto store = [&](int c, const uint32_t (&x)[32]) {
                if (mine(tile) && m0 + c * 32 < end) pt_store(job, row, m0 + c * 32, end, x);
            };
            // columns past the tile's are not stored
            pg_tmem_ld32(lanes + (uint32_t)(grp * 32), v[0]);
            if (parts == 2) {
                store(grp, v[0]);
                pg_tmem_ld32(lanes + (uint32_t)((grp + 8) * 32), v[0]);
            }
            pg_tmem_ld32(lanes + (uint32_t)((grp + 4) * 32), v[1]);
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pt_arrive_shared(ps_map(smem_u32(&acc_free), even));
            store(parts == 2 ? grp + 8 : grp, v[0]);
            store(grp + 4, v[1]);
        };
        auto hand_over = [&](uint32_t stage) {
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pt_arrive_shared(ps_map(smem_u32(&w_full[stage]), even));
        };
        // one more pass than there are tiles: the last one only finishes the tile before it
        int count = 0;
        for (int tile = pair0; ok; tile += n_pairs, count++) {
            const bool more = tile < P.tiles;
            if (!more && (CUT || count == 0)) break;
            int local;
            const int js = job_of(min(tile, P.tiles - 1), local);
            const PgJob &job = jobs.j[js];
            const bool q4 = job.type == TYPE_Q4_K, pair = job.w2 != nullptr, skew = (P.skew >> js) & 1;
            const int row = pt_row(pair, skew, q);
            const uint8_t *at = smem + PT_RING + (uint32_t)pt_place(pair, skew, row) * (q4 ? PT_Q4_PITCH : PT_Q6_PITCH);
            // Q6_K: bytes from the last 16-byte boundary to the row's next block
            uint32_t shift = (uint32_t)b0 * Q6K_BYTES;
            if (skew) shift += (uint32_t)((uintptr_t)(pair && lane >= 16 ? job.w2 : job.w) + (uint32_t)(row & 7) * (uint32_t)nb_row * Q6K_BYTES) & 15u;
            for (int b = 0; b < nb; b++, shift += Q6K_BYTES) {
                if (more) {
                    uint32_t o[32];
                    ok = pt_warp_wait(&raw_full[rs], rphase);
                    if (!ok) break;
                    auto read = [&]() {
                        __syncwarp();
                        if (lane == 0) pg_arrive(&raw_empty[rs]);
                    };
                    // an infinite scale of a Q6_K block (the look for one costs 0.7 % of a 203-token prompt)
                    auto beyond = [&]() { return (*reinterpret_cast<const uint16_t *>(at + rs * PT_RAW_BYTES + (shift & 15u) + 208) & 0x7c00u) == 0x7c00u; };
                    if (q4) pt_dequant_q4(at + rs * PT_RAW_BYTES, grp, o, read);
                    else if (skew || __any_sync(0xffffffffu, beyond())) pt_dequant_q6(at + rs * PT_RAW_BYTES + (shift & 15u), grp, o, read);
                    else {
                        const uint8_t *base = at + rs * PT_RAW_BYTES;
                        const uint32_t odd = (shift >> 1) & 1u;
                        switch ((shift >> 2) & 3u) {
                        case 0: pt_dequant_q6_at<0>(base, odd, grp, o, read); break;
                        case 1: pt_dequant_q6_at<1>(base, odd, grp, o, read); break;
                        case 2: pt_dequant_q6_at<2>(base, odd, grp, o, read); break;
                        default: pt_dequant_q6_at<3>(base, odd, grp, o, read); break;
                        }
                    }
                    if (++rs == PT_RAWS) rs = 0, rphase ^= 1u;
                    const uint32_t s = (parts == 2 ? 0u : 2u * (uses & 1u)) + (uint32_t)(grp >> 1);
                    ok = pt_warp_wait(&empty[s], ((uses >> (ring_log - 1)) & 1u) ^ 1u);
                    if (!ok) break;
                    pg_fence_after();
                    pt_tmem_st32(lanes + w_col + 64u * s + 32u * (uint32_t)(grp & 1), o);
                    hand_over(s);
                    uses++;
                }
                if (!CUT && b == 0 && count > 0) {
                    pdl_wait();   // stores come after the launches before this one
                    finish(tile - n_pairs, count - 1);
                }
                if (!more || !ok) break;
            }
            if (!more) break;
        }
    } else if (warp == PT_WORKERS) {
        if (rank == 0) {
            if (pg_elect()) {
                const uint32_t idesc = pt_idesc(part);
                uint32_t s = 0, phase = 0;
                int count = 0;
                for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs, count++) {
                    if (count > 0) ok = pt_wait(&acc_free, (uint32_t)((count - 1) & 1));
                    for (int kt = 0; kt < 2 * nb && ok; kt++) {
                        ok = pt_wait_shared(&full[s], &w_full[s], phase);
                        if (!ok) break;
                        pg_fence_after();
                        const uint64_t dx = pg_smem_desc(smem_u32(smem + s * stage_bytes));
                        const uint32_t w = tmem + w_col + 64u * s;
#pragma unroll
                        for (int k = 0; k < 8; k++) pt_mma(tmem, w + 8u * k, dx + (k >= 4 ? panel >> 4 : 0u) + 2u * (k & 3), idesc, (kt | k) != 0);   // 32 bytes on
                        if (parts == 2) {
#pragma unroll
                            for (int k = 0; k < 8; k++)
                                pt_mma(tmem + (uint32_t)part, w + 8u * k, dx + (half_bytes >> 4) + (k >= 4 ? panel >> 4 : 0u) + 2u * (k & 3), idesc, (kt | k) != 0);
                        }
                        pt_commit(&empty[s], even);
                        if (++s == ring) s = 0, phase ^= 1u;
                    }
                    if (ok) pt_commit(&acc_full, even);
                }
            }
        }
        __syncwarp();
    } else if (warp == PT_WORKERS + 1) {
        if (lane == 0) {
            pdl_wait();   // the tokens are the previous launch's result
            uint32_t st = 0;
            for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs) {
                const int m0 = (tile % P.token_tiles) * P.nt + rank * (part / 2);
                for (int kt = 0; kt < 2 * nb; kt++, st++) {
                    const uint32_t s = st & (ring - 1), to = smem_u32(smem + s * stage_bytes), bar = ps_map(smem_u32(&full[s]), even);
                    ok = mbar_wait_bounded(&empty[s], ((st >> ring_log) & 1u) ^ 1u);
                    if (!ok) break;
                    if (rank == 0) mbar_arrive_expect_tx(&full[s], 2 * stage_bytes);   // both CTAs' copies
                    for (uint32_t i = 0; i < 2; i++)
                        for (int j = 0; j < parts; j++) pt_tma_2d(to + i * panel + (uint32_t)j * half_bytes, &maps.x, (4 * b0 + 2 * kt + (int)i) * PG_K, m0 + j * part, bar);
                }
            }
            ps_st_remote(ps_map(smem_u32(&s_issued[rank]), even), st);
        }
    } else if (lane == 0) {
        // blocks of K as they are in memory
        uint32_t raws = 0;
        for (int tile = pair0; tile < P.tiles && ok; tile += n_pairs) {
            int local;
            const int js = job_of(tile, local);
            const PgJob &job = jobs.j[js];
            const bool q4 = job.type == TYPE_Q4_K, skew = (P.skew >> js) & 1;
            const uint32_t pitch = q4 ? PT_Q4_PITCH : PT_Q6_PITCH, row_bytes = (uint32_t)nb_row * Q6K_BYTES;
            const int y = local * (job.w2 ? PG_ROWS / 2 : PG_ROWS);
            for (int b = b0; b < b0 + nb; b++, raws++) {
                const uint32_t s = raws % PT_RAWS, to = smem_u32(smem + PT_RING + s * PT_RAW_BYTES);
                ok = mbar_wait_bounded(&raw_empty[s], ((raws / PT_RAWS) & 1u) ^ 1u);
                if (!ok) break;
                mbar_arrive_expect_tx(&raw_full[s], PG_ROWS * pitch);
                // x: 8-byte words, even: a 16-byte boundary
                if (skew) {
                    const uint32_t box = (job.w2 ? 8 : 16) * PT_Q6_PITCH;
                    for (uint32_t j = 0; j < 8; j++) {
                        const uint32_t at = j * row_bytes, off = (uint32_t)b * Q6K_BYTES;
                        pg_tma_2d(to + j * box, &maps.w[js][j], (int)((((uint32_t)(uintptr_t)job.w + at & 15u) + off) / 16 * 2), y >> 3, &raw_full[s]);
                        if (job.w2) pg_tma_2d(to + (8 + j) * box, &maps.w2[j], (int)((((uint32_t)(uintptr_t)job.w2 + at & 15u) + off) / 16 * 2), y >> 3, &raw_full[s]);
                    }
                } else {
                    const int x = q4 ? b * (int)(Q4K_BYTES / 8) : b * (int)Q6K_BYTES / 16 * 2;
                    pg_tma_2d(to, maps.w[js], x, y, &raw_full[s]);
                    pg_tma_2d(to + PG_ROWS / 2 * pitch, job.w2 ? maps.w2 : maps.w[js], x, job.w2 ? y : y + PG_ROWS / 2, &raw_full[s]);
                }
            }
        }
        pg_drain(raw_full, raws, PT_RAWS);
    }
    if (!ok) s_failed = 1;
    __syncwarp();
    if constexpr (CUT) {
        __syncthreads();   // a failure of any role
        pdl_wait();        // every thread that stores comes after the launches before this one
        bool fin = s_failed == 0;
        fin = __all_sync(0xffffffffu, fin && mbar_wait_bounded(&acc_full, 0u));
        if (!fin) s_failed = 1;
        pg_fence_after();
        ps_cluster_sync();   // every CTA's MMAs have read their tokens: the slots may be written
        int local;
        const PgJob &job = jobs.j[job_of(pair0, local)];
        const int row = row_of(pair0), m0 = (pair0 % P.token_tiles) * P.nt, end = min(P.seq, m0 + P.nt);
        const bool store = fin && mine(pair0);
        ps_reduce<8, 4, PT_RING>(ks, kr, (end - m0 + 31) / 32, smem, tmem, warp < PT_WORKERS, q, grp, fin, [&](int cc, int, const float (&sum)[8]) {
            uint32_t v[8];
#pragma unroll
            for (int t = 0; t < 8; t++) v[t] = __float_as_uint(sum[t]);
            if (store) pt_store(job, row, m0 + cc * 32 + grp * 8, end, v);
        }, 2, rank);
    }
    pg_fence_before();
    __syncthreads();
    ps_cluster_sync();   // the other CTAs' memory and barriers are no longer used
    if (s_failed) {
        // Accumulators that are complete mean that all copies have landed.  Who gave up does not know: both CTAs' token copies count on
        // the even CTA's barriers, and what the odd one asked for beyond the even one's last stage is announced here.  The odd CTA
        // stays for it if it has given up too.
        if (rank == 0 && tid == 0) {
            for (uint32_t i = s_issued[0]; i < s_issued[1]; i++) mbar_arrive_expect_tx(&full[i & (ring - 1)], 2 * stage_bytes);
            pg_drain(full, max(s_issued[0], s_issued[1]), ring);
        }
        __syncthreads();
        ps_cluster_sync();
    }
    if (warp == PT_WORKERS) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
        if (lane == 0 && s_failed && err_flag) atomicExch(err_flag, DEV_ERR_GEMM_TIMEOUT);
    }
}

}  // namespace rnb
