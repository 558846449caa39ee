// Prefill matmul on the 5th-generation tensor cores: Y[t][row] = sum_k W[row][k] * X[t][k] for a
// batch of tokens, W in GGUF Q4_K / Q6_K blocks, dequantised tile-wise to bf16 in shared
// memory and multiplied with tcgen05.mma (bf16 x bf16 -> fp32 accumulators in tensor memory).
// Replaces the reference's dequant -> f16 + cublasGemmEx path (q4k_f16_gemm_batch,
// crates/rnb-backend/cuda/src/runtime/gemv.rs:2335-2421); the dequantisation follows
// crates/rnb-cpu/src/quantize/dequant.rs:353-381 (Q4_K) and :780-807 (Q6_K) in f32 and rounds
// once to bf16.
//
// What the three kernels share (prefill_gemm_pair.cuh: pairs of SMs, weights in tensor memory; prefill_gemm_wide.cuh: pairs of SMs, tiles of
// up to 512 tokens, weights in shared memory; prefill_gemm_split.cuh: a few tokens of short rows, the same): the weight tile is the M operand (tensor-memory lane = weight row), the tokens the N
// operand.  Operand tiles in shared memory are 64 elements of K, K-major in the 128-byte swizzle the MMA descriptors expect:
//   byte offset of (row r, 16-byte chunk c) = (r / 8) * 1024 + (r % 8) * 128 + ((c ^ (r % 8)) * 16).
// Tokens come in by tiled TMA copies (rows past the end of the batch read as zeros).  Every wait is bounded; a
// timeout sets the error flag and all roles still meet at the final barrier, where the tensor memory is freed.
#pragma once
#include <cuda_bf16.h>

#include <type_traits>

#include "bounded_walk.hpp"
#include "common.cuh"

namespace rnb {

constexpr int PG_ROWS = 128;     // weight rows per CTA
constexpr int PG_K = 64;         // elements per stage
constexpr uint32_t PG_B_BYTES = PG_ROWS * 128;   // weight tile of a stage

// K-major, 128-byte swizzle, 8-row groups 1024 bytes apart; descriptor version 1 (sm_100)
__device__ __forceinline__ uint64_t pg_smem_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// One lane of a converged warp.  The MMAs are issued behind this and not behind `lane == 0`, where a stage of eight took 1000
// cycles to issue (clock64 around it).
__device__ __forceinline__ bool pg_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void pg_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void pg_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pg_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pg_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void pg_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// The copies that a producer announced on a ring of barriers have landed (bounded, as every wait).
__device__ __forceinline__ void pg_drain(uint64_t *full, uint32_t issued, uint32_t ring) {
    drain_ring(issued, ring, [&](uint32_t slot, uint32_t parity) {
        for (uint32_t k = 0; k < (1u << 18) && !mbar_try_wait(&full[slot], parity); k++) {
            if (k > 64) __nanosleep(64);
        }
    });
}
__device__ __forceinline__ void pg_tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
          "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]),
          "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
          "=r"(v[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// q in 0..255 -> exact f32 without an int-to-float conversion: the bits of 2^23 + q, minus 2^23 (Q6_K: minus 2^23 + 32);
// two of them at a time as packed f32: ((2^23 + q) - 2^23) * s + m of bytes b and b + 1 of `word`, rounded to a bf16 pair.  The
// same roundings as one by one, five instructions for two elements instead of seven.
__device__ __forceinline__ uint64_t pg_pair_f32(float a, float b) { return (uint64_t)__float_as_uint(a) | (uint64_t)__float_as_uint(b) << 32; }
__device__ __forceinline__ uint32_t pg_dequant_pair_fma(uint32_t word, int b, uint64_t s, uint64_t m) {
    uint32_t r;
    asm("{\n\t.reg .b64 t;\n\t.reg .b32 x, y;\n\tmov.b64 t, {%1, %2};\n\tadd.rn.f32x2 t, t, %3;\n\tfma.rn.f32x2 t, t, %4, %5;\n\tmov.b64 {x, y}, t;\n\t"
        "cvt.rn.bf16x2.f32 %0, y, x;\n\t}"
        : "=r"(r)
        : "r"(__byte_perm(word, 0x4b000000u, 0x7650 + b)), "r"(__byte_perm(word, 0x4b000000u, 0x7651 + b)), "l"(0xcb000000cb000000ull), "l"(s), "l"(m));
    return r;
}
__device__ __forceinline__ uint32_t pg_dequant_pair_mul_m32(uint32_t word, int b, uint64_t s) {   // (q - 32) * s
    uint32_t r;
    asm("{\n\t.reg .b64 t;\n\t.reg .b32 x, y;\n\tmov.b64 t, {%1, %2};\n\tadd.rn.f32x2 t, t, %3;\n\tmul.rn.f32x2 t, t, %4;\n\tmov.b64 {x, y}, t;\n\t"
        "cvt.rn.bf16x2.f32 %0, y, x;\n\t}"
        : "=r"(r)
        : "r"(__byte_perm(word, 0x4b000000u, 0x7650 + b)), "r"(__byte_perm(word, 0x4b000000u, 0x7651 + b)), "l"(0xcb000020cb000020ull), "l"(s));
    return r;
}
__device__ __forceinline__ uint32_t pg_pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// ---- raw bytes of a weight group (64 elements of one row) --------------------------------------
// The two threads of a row fetch disjoint halves of what both need (the block header once per
// block, the group's 32 qs bytes every stage) and exchange them by shuffle when the bytes are
// used: every byte of a weight tile crosses the L2 -> SM path once.
__device__ __forceinline__ uint4 pg_pair_exchange(const uint4 &mine) {
    return make_uint4(__shfl_xor_sync(0xffffffffu, mine.x, 1), __shfl_xor_sync(0xffffffffu, mine.y, 1), __shfl_xor_sync(0xffffffffu, mine.z, 1),
                      __shfl_xor_sync(0xffffffffu, mine.w, 1));
}
// f32 -> bf16 rows (activation), padded to a multiple of 8 columns by construction (cols % 256 == 0)
RNB_GLOBAL void __launch_bounds__(256)
f32_to_bf16_kernel(const float *x, uint16_t *y, size_t n) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= n) return;
    const float4 a = *reinterpret_cast<const float4 *>(x + i), b = *reinterpret_cast<const float4 *>(x + i + 4);
    *reinterpret_cast<uint4 *>(y + i) = make_uint4(pg_pack_bf16(a.x, a.y), pg_pack_bf16(a.z, a.w), pg_pack_bf16(b.x, b.y), pg_pack_bf16(b.z, b.w));
}

// Residual add + RMSNorm of a batch of token rows, written straight as the bf16 token matrix of
// the next matmul: x += t (when t is given; x is updated in place), then (x / rms) * w with the
// f64 mean square of rnb-cpu's rms_norm_into (crates/rnb-cpu/src/kernels/norm.rs:177-196), rounded once to bf16.  One CTA per
// token; hidden % 256 == 0.  A row of up to 16 elements per thread stays in registers between the sum and the output.
template <int THREADS>
RNB_GLOBAL void __launch_bounds__(THREADS)
add_rmsnorm_bf16_kernel(float *x, const float *t, const float *__restrict__ w, float eps, int hidden,
                        uint16_t *out) {
    constexpr int KEEP = 4;
    pdl_launch_dependents();
    pdl_wait();
    __shared__ double red[THREADS / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n4 = hidden / 4;
    float4 *xs = reinterpret_cast<float4 *>(x + (size_t)blockIdx.x * hidden);
    const float4 *ts = t ? reinterpret_cast<const float4 *>(t + (size_t)blockIdx.x * hidden) : nullptr;
    double ss = 0.0;
    float4 keep[KEEP];
    auto take = [&](int i) {
        float4 v = xs[i];
        if (ts) {
            const float4 a = ts[i];
            v = make_float4(__fadd_rn(v.x, a.x), __fadd_rn(v.y, a.y), __fadd_rn(v.z, a.z), __fadd_rn(v.w, a.w));
            xs[i] = v;
        }
        ss += ((double)v.x * v.x + (double)v.y * v.y) + ((double)v.z * v.z + (double)v.w * v.w);
        return v;
    };
#pragma unroll
    for (int k = 0; k < KEEP; k++)
        if (tid + k * THREADS < n4) keep[k] = take(tid + k * THREADS);
    for (int i = tid + KEEP * THREADS; i < n4; i += THREADS) take(i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    double a = 0.0;
    for (int i = 0; i < THREADS / 32; i++) a += red[i];
    const float rms = (float)sqrt(a / (double)hidden + (double)eps);
    uint2 *os = reinterpret_cast<uint2 *>(out + (size_t)blockIdx.x * hidden);
    const float4 *ws = reinterpret_cast<const float4 *>(w);
    auto put = [&](int i, const float4 &v) {
        const float4 g = ws[i];
        os[i] = make_uint2(pg_pack_bf16(__fmul_rn(__fdiv_rn(v.x, rms), g.x), __fmul_rn(__fdiv_rn(v.y, rms), g.y)),
                           pg_pack_bf16(__fmul_rn(__fdiv_rn(v.z, rms), g.z), __fmul_rn(__fdiv_rn(v.w, rms), g.w)));
    };
#pragma unroll
    for (int k = 0; k < KEEP; k++)
        if (tid + k * THREADS < n4) put(tid + k * THREADS, keep[k]);
    for (int i = tid + KEEP * THREADS; i < n4; i += THREADS) put(i, xs[i]);   // this thread's own stores
}

// silu(gate) * up (g / (1 + exp(-g)), crates/rnb-cpu/src/kernels/activation.rs:74-89, libm's expf as in
// silu_mul_q8k_kernel) written straight as the bf16 token matrix of the down
// matmul: the f32 value is rounded to bf16 exactly as f32_to_bf16_kernel would round it.
RNB_GLOBAL void __launch_bounds__(256)
silu_mul_bf16_kernel(const float *gate, const float *up, uint16_t *y, size_t n) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i >= n) return;
    const float4 g0 = *reinterpret_cast<const float4 *>(gate + i), g1 = *reinterpret_cast<const float4 *>(gate + i + 4);
    const float4 u0 = *reinterpret_cast<const float4 *>(up + i), u1 = *reinterpret_cast<const float4 *>(up + i + 4);
    const float gv[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, uv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float e = expf_libm(-gv[j]);
        v[j] = __fmul_rn(__fdiv_rn(gv[j], __fadd_rn(1.0f, e)), uv[j]);
    }
    *reinterpret_cast<uint4 *>(y + i) = make_uint4(pg_pack_bf16(v[0], v[1]), pg_pack_bf16(v[2], v[3]), pg_pack_bf16(v[4], v[5]), pg_pack_bf16(v[6], v[7]));
}

// 128-byte, 64-byte aligned descriptor of the bf16 token matrix [seq][cols] (a CUtensorMap, kept
// opaque here): boxes of 64 columns x as many rows as the kernel asks for, 128-byte swizzle, zero fill past the end.
struct alignas(64) PgTensorMap {
    unsigned long long opaque[16];
};
// tiled 2-D copy global -> shared; x (elements of the inner dimension) * 2 bytes must be a multiple of 16
__device__ __forceinline__ void pg_tma_2d(uint32_t dst, const void *tmap, int x, int y, uint64_t *bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(tmap), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

// Up to three matrices that share the token tile go out in one launch (q/k/v, gate/up): the
// row tiles of all of them are numbered through.
constexpr int PG_MAX_JOBS = 3;
struct PgJob {
    const uint8_t *w;
    float *y;     // [seq][rows]
    int rows, type, tile0, pad;
    // gate + up form (w2 != null): a tile is 64 rows of w (gate) and the same 64 rows of w2 (up); the epilogue writes
    // silu(gate) * up as bf16 [seq][rows] to yb - the token matrix of the down matmul
    const uint8_t *w2;
    uint16_t *yb;
};
struct PgJobs {
    PgJob j[PG_MAX_JOBS];
    int n;
};

// Half h of a Q4_K group: h = 0 -> low nibbles (chunks 0-3), h = 1 -> high nibbles (chunks 4-7).
// y = (d*sc)*q - (dmin*m) (crates/rnb-cpu/src/quantize/dequant.rs:353-381), evaluated with one fused
// multiply-add per element: the f32 value can differ from the two-rounding form in its last bit,
// which survives the rounding to bf16 only next to a tie.
__device__ __forceinline__ void pg_dequant_q4(const uint4 &hdr, const uint4 &q0, const uint4 &q1, int g, int h, uint8_t *row_base, int rr) {
    const float d = f16_bits_to_f32(hdr.x & 0xffffu), dmin = f16_bits_to_f32(hdr.x >> 16);
    const uint32_t sc03 = hdr.y & 0x3f3f3f3fu, mn03 = hdr.z & 0x3f3f3f3fu;
    const uint32_t sc47 = (hdr.w & 0x0f0f0f0fu) | (((hdr.y >> 6) & 0x03030303u) << 4);
    const uint32_t mn47 = ((hdr.w >> 4) & 0x0f0f0f0fu) | (((hdr.z >> 6) & 0x03030303u) << 4);
    const uint32_t scw = g < 2 ? sc03 : sc47, mnw = g < 2 ? mn03 : mn47;
    const int sh = 16 * (g & 1) + 8 * h;
    const float ds = __fmul_rn(d, (float)((scw >> sh) & 0xffu)), nm = -__fmul_rn(dmin, (float)((mnw >> sh) & 0xffu));
    const uint64_t ds2 = pg_pair_f32(ds, ds), nm2 = pg_pair_f32(nm, nm);
    const uint32_t qw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    const int nsh = 4 * h;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        uint32_t o[4];
#pragma unroll
        for (int w = 0; w < 2; w++) {
            const uint32_t n4 = (qw[2 * c + w] >> nsh) & 0x0f0f0f0fu;
            o[2 * w] = pg_dequant_pair_fma(n4, 0, ds2, nm2);
            o[2 * w + 1] = pg_dequant_pair_fma(n4, 2, ds2, nm2);
        }
        *reinterpret_cast<uint4 *>(row_base + (((c + 4 * h) ^ rr) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}
// Q6_K: group g of a block = elements 64g..64g+63 = for half n = g/2 the pair (q1,q2) if g even,
// (q3,q4) if g odd, l = 0..31 each; y = (d*sc)*(q-32): dequant.rs:780-807.  Blocks are 210 bytes,
// so rows are only 2-byte aligned: bytes are fetched as aligned 16-byte windows and shifted into place (pg_ldg_window).
// Half h of the Q6_K groups of half-block n: h = 0 -> ql[64n .. 64n+31] (q1 / q3), h = 1 -> ql[64n+32 ..] (q2 / q4).
struct PgRawQ6 {
    uint32_t ql[8], qh[4];   // qh: words 4h .. 4h+3 of the half-block's 32 bytes, the pair exchanges them when used
    uint32_t sc[2];
    float d;
};
// NW consecutive words from a 2-byte aligned address out of NV aligned 16-byte loads (4 NV >= NW + 4): the words of the
// loaded window are shifted by whole words with two levels of selects, then funnel-shifted by the odd half-word.  The
// threads of a warp read rows that lie kilobytes apart, so every load instruction costs 32 cache-line accesses
// whatever its width: seven 16-byte loads per half block instead of eighteen 4-byte ones is what lifts the Q6_K
// producer off the load pipe.  An aligned 16-byte load that contains one byte of the tensor cannot leave its page.
template <int NW, int NV, bool SHARED = false>
__device__ __forceinline__ void pg_ldg_window(const uint8_t *p, uint32_t *out, uint32_t *raw = nullptr) {
    static_assert(4 * NV >= NW + 4, "window too small");
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    const uint8_t *base = p - (a & 15);
    const uint32_t off = (uint32_t)(a & 15), k = off >> 2, sh = (off & 3u) * 8u;
    uint32_t v[4 * NV];
#pragma unroll
    for (int j = 0; j < NV; j++) {
        uint4 t;
        if constexpr (SHARED) t = *reinterpret_cast<const uint4 *>(base + 16 * j);
        else t = ldg_nc_u4(base + 16 * j);
        v[4 * j] = t.x, v[4 * j + 1] = t.y, v[4 * j + 2] = t.z, v[4 * j + 3] = t.w;
    }
    if (raw) {
#pragma unroll
        for (int i = 0; i < 4 * NV; i++) raw[i] = v[i];
    }
    uint32_t s1[NW + 2], s2[NW + 1];
#pragma unroll
    for (int i = 0; i < NW + 2; i++) s1[i] = (k & 2u) ? v[i + 2] : v[i];
#pragma unroll
    for (int i = 0; i < NW + 1; i++) s2[i] = (k & 1u) ? s1[i + 1] : s1[i];
#pragma unroll
    for (int i = 0; i < NW; i++) out[i] = __funnelshift_r(s2[i], s2[i + 1], sh);
}
__device__ __forceinline__ void pg_load_q6(PgRawQ6 &r, const uint8_t *blk, int n, int h) {
    pg_ldg_window<8, 3>(blk + 64 * n + 32 * h, r.ql);
    pg_ldg_window<4, 2>(blk + 128 + 32 * n + 16 * h, r.qh);
    // scales (16 bytes at 192) and d (2 bytes at 208): one 18-byte window = two aligned 16-byte loads
    uint32_t sc4[4], raw[8];
    pg_ldg_window<4, 2>(blk + 192, sc4, raw);
    r.sc[0] = n ? sc4[2] : sc4[0];
    r.sc[1] = n ? sc4[3] : sc4[1];
    // d sits 16 bytes after the window's first byte: in the second 16-byte load, at the same offset
    const uint32_t dpos = (uint32_t)(reinterpret_cast<uintptr_t>(blk + 192) & 15u), dk = dpos >> 2;
    const uint32_t dlo = (dk & 2u) ? ((dk & 1u) ? raw[7] : raw[6]) : ((dk & 1u) ? raw[5] : raw[4]);
    r.d = f16_bits_to_f32((dlo >> ((dpos & 2u) * 8u)) & 0xffffu);
}
// ql, qh: this half's 32 low and high bytes; scw: its two scale bytes
__device__ __forceinline__ void pg_dequant_q6_half(const uint32_t (&ql)[8], const uint32_t (&qh)[8], uint32_t scw, float d, bool odd, int h, uint8_t *row_base, int rr) {
    const float ds0 = __fmul_rn(d, (float)(int)(int8_t)(scw & 0xffu)), ds1 = __fmul_rn(d, (float)(int)(int8_t)((scw >> 8) & 0xffu));
    const uint64_t sp[2] = {pg_pair_f32(ds0, ds0), pg_pair_f32(ds1, ds1)};
    // the two high bits of this half's elements sit at bit 2h (even group) or 4 + 2h (odd group) of qh
    const int hs = (odd ? 4 : 0) + 2 * h, ls = odd ? 4 : 0;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        uint32_t o[4];
#pragma unroll
        for (int w = 0; w < 2; w++) {
            const int i = 2 * c + w;
            const uint32_t q = ((ql[i] >> ls) & 0x0f0f0f0fu) | (((qh[i] >> hs) << 4) & 0x30303030u);
            o[2 * w] = pg_dequant_pair_mul_m32(q, 0, sp[c >> 1]);
            o[2 * w + 1] = pg_dequant_pair_mul_m32(q, 2, sp[c >> 1]);
        }
        *reinterpret_cast<uint4 *>(row_base + (((c + 4 * h) ^ rr) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
}
__device__ __forceinline__ void pg_dequant_q6(const PgRawQ6 &r, int g, int h, uint8_t *row_base, int rr) {
    const bool odd = g & 1;
    uint32_t qh[8];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, r.qh[i], 1);
        qh[i] = h ? other : r.qh[i];
        qh[4 + i] = h ? r.qh[i] : other;
    }
    pg_dequant_q6_half(r.ql, qh, (odd ? r.sc[1] : r.sc[0]) >> (16 * h), r.d, odd, h, row_base, rr);
}

}  // namespace rnb
