"""Prefill matmul of short prompts (K cut over a cluster): token counts at the edges of the tiles, ragged rows, and
blocks of K that do not divide evenly, against the oracle's weights and the tokens, both rounded once to bf16, in f64.

Bound: f32 accumulation only, a random walk of sqrt(K) * 2^-24 of the dot product's scale sqrt(sum (x w)^2) per
partial sum (under 1e-5 at K = 14336); 1e-4 of that scale, as for the 512-token tiles."""
import numpy as np
import pytest

import oracle as orc
from synth import Q4_K, Q6_K, quantized, random_blocks
from test_gpu_prefill_gemm import bf16_round, ops  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,rows,cols,seq", [
    (Q4_K, 128, 256, 1), (Q4_K, 129, 768, 16), (Q6_K, 127, 512, 17), (Q4_K, 200, 1024, 255), (Q6_K, 130, 1280, 256), (Q4_K, 256, 2304, 257),
    (Q6_K, 100, 2048, 290), (Q4_K, 260, 4096, 33), (Q6_K, 256, 8448, 48), (Q4_K, 128, 14336, 300), (Q6_K, 384, 14336, 511), (Q4_K, 64, 8192, 511),
    (Q4_K, 9700, 1024, 1), (Q6_K, 9700, 1024, 17), (Q4_K, 200, 1024, 128), (Q4_K, 19000, 256, 64), (Q4_K, 19000, 512, 128), (Q6_K, 100, 2048, 129),
])
def test_short_prompt_matmul(ops, t, rows, cols, seq):
    rng = np.random.default_rng(rows + 7 * cols + seq)
    w = quantized(rng, t, rows, cols)[1] if rows * cols < 1 << 20 else random_blocks(rng, t, rows, cols)
    x = rng.standard_normal((seq, cols)).astype(np.float32)
    wd = orc.dequantize_matrix(t, w, rows, cols).reshape(rows, cols)
    fn = ops.q4k_bf16_gemm_batch if t == Q4_K else ops.q6k_bf16_gemm_batch
    got = fn(w, rows, cols, x).reshape(seq, rows)
    ref = bf16_round(x).astype(np.float64) @ bf16_round(wd).astype(np.float64).T
    scale = np.sqrt((x.astype(np.float64) ** 2) @ (wd.astype(np.float64) ** 2).T)
    assert np.max(np.abs(got - ref) / np.maximum(scale, 1e-30)) <= 1e-4
    assert np.array_equal(got, fn(w, rows, cols, x).reshape(seq, rows))   # summed in rank order: the same bits each time


@pytest.mark.parametrize("t,rows,cols,seq", [(Q4_K, 64, 1024, 16), (Q4_K, 1000, 2048, 45), (Q6_K, 65, 768, 256), (Q4_K, 4096, 1024, 255)])
def test_short_prompt_gate_up(ops, t, rows, cols, seq):
    """silu(gate) * up as bf16: half an ulp (2^-8 at most) of the result, plus what f32 sums in another order move g and
    u by (1e-4 of their scale, as above), relative to the largest result."""
    import torch

    import runnburn_b200 as r
    rng = np.random.default_rng(rows + seq)
    ws = [quantized(rng, t, rows, cols)[1] for _ in range(2)]
    x = rng.standard_normal((seq, cols)).astype(np.float32)
    g, u = (bf16_round(x).astype(np.float64) @ bf16_round(orc.dequantize_matrix(t, w, rows, cols).reshape(rows, cols)).astype(np.float64).T for w in ws)
    ref = g / (1.0 + np.exp(-g)) * u
    wt, xt = [torch.from_numpy(np.ascontiguousarray(w)).cuda() for w in ws], torch.from_numpy(x).cuda()
    xb = torch.empty(seq * cols, dtype=torch.int16, device="cuda")
    act = torch.zeros(seq, rows, dtype=torch.bfloat16, device="cuda")
    assert r.load().rnb_b200_dev_prefill_gemm_silu(t, wt[0].data_ptr(), wt[1].data_ptr(), rows, cols, xt.data_ptr(), seq, xb.data_ptr(), act.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert ops.dev_error_flag() == 0
    got = act.float().cpu().numpy().astype(np.float64)
    assert np.max(np.abs(got - ref) - 2.0 ** -8 * np.abs(ref)) <= 1e-4 * np.max(np.abs(ref))


@pytest.mark.parametrize("n", [9, 16, 17, 128, 129, 256, 257, 300])
@pytest.mark.parametrize("design", ["dutivik", "punisun"])
def test_prompt_products_cut_along_k(design, n):
    """bf16 stacks whose products have 16 to 48 stages of K and few tiles (4 or 8 CTAs along K; the gate and up pair too, but for
    257 and 300 tokens, where pairs of SMs take it), at the edges of the token tiles, against the plain reference: every
    projection rounds its input to bf16, the bound of the stack tests (3e-2 of the rows' scale)."""
    import stack_util as su
    from hybrid_ref import Model
    if design == "dutivik":
        cfg = su.dutivik([su.gla(heads=4, dim=64, vdim=64, ff=2816)], width=1024)
    else:
        cfg = su.config([su.retention(heads=4, dim=64, vdim=64, ff=1920)], width=1024)
    w = su.weights(cfg, seed=n, rank=16)
    toks = su.tokens(cfg, n, seed=1)
    dec = su.decoder(cfg, w, "bfloat16", max_ctx=512)
    want = Model(cfg, w).forward(toks)
    got = dec.prefill_logits(toks, 0, list(range(n)))[0]
    dec.close()
    assert not (why := su.bad(got, want, "bfloat16")), why


@pytest.mark.parametrize("specs,cols,seq", [
    ([(Q4_K, 9600)], 1024, 128), ([(Q4_K, 19000)], 1024, 128), ([(Q4_K, 19000)], 1024, 129), ([(Q6_K, 19000)], 1024, 65), ([(Q4_K, 4700), (Q6_K, 4700)], 2048, 300),
    ([(Q4_K, 2500)] * 3, 2048, 511), ([(Q6_K, 300)], 1024, 129), ([(Q4_K, 300)], 3840, 129), ([(Q4_K, 4800)], 8192, 257), ([(Q4_K, 300)], 768, 64), ([(Q4_K, 300)], 768, 65),
])
def test_launches_that_fill_the_chip_are_not_cut(ops, specs, cols, seq):
    """A launch whose tiles fill the chip, or whose rows are short, sums a token's products in one chain along K, as a prompt of 600
    tokens does: the same bits for the tokens that they share."""
    import ctypes

    import torch

    import runnburn_b200 as r
    rng = np.random.default_rng(cols + seq)
    n = len(specs)
    w = [torch.from_numpy(random_blocks(rng, t, rows, cols)).cuda() for t, rows in specs]
    x = torch.randn(600, cols, device="cuda", generator=torch.Generator("cuda").manual_seed(seq))
    xb = torch.empty(600 * cols, dtype=torch.int16, device="cuda")
    out = {}
    for tokens in (seq, 600):
        ys = [torch.full((tokens, rows), float("nan"), device="cuda") for _, rows in specs]
        assert r.load().rnb_b200_dev_prefill_gemm_multi(
            n, (ctypes.c_int * n)(*[t for t, _ in specs]), (ctypes.c_void_p * n)(*[v.data_ptr() for v in w]), (ctypes.c_size_t * n)(*[rows for _, rows in specs]),
            (ctypes.c_void_p * n)(*[y.data_ptr() for y in ys]), cols, x.data_ptr(), tokens, xb.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert ops.dev_error_flag() == 0
        out[tokens] = ys
    for a, b in zip(out[seq], out[600]):
        assert torch.equal(a, b[:seq])
