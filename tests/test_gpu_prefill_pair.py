"""Prefill matmul of long prompts (pairs of SMs): odd numbers of row tiles, ragged rows and tokens, one block of K, pairs
that take several tiles in turn, rows that tiled copies cannot describe (Q6_K, a number of blocks that is not a multiple
of eight), and matrices of both formats in one launch, against the oracle's weights and the tokens, both rounded once to
bf16, in f64.

Bound: f32 accumulation only, 1e-4 of a dot product's scale sqrt(sum (x w)^2), as for the other prompt kernels."""
import ctypes

import numpy as np
import pytest

import oracle as orc
from synth import Q4_K, Q6_K, quantized, random_blocks
from test_gpu_prefill_gemm import bf16_round, ops  # noqa: F401

pytestmark = pytest.mark.gpu


def weights(rng, t, rows, cols):
    return quantized(rng, t, rows, cols)[1] if rows * cols < 1 << 20 else random_blocks(rng, t, rows, cols)


def off(got, t, w, rows, cols, x):
    wd = orc.dequantize_matrix(t, w, rows, cols).reshape(rows, cols)
    ref = bf16_round(x).astype(np.float64) @ bf16_round(wd).astype(np.float64).T
    scale = np.sqrt((x.astype(np.float64) ** 2) @ (wd.astype(np.float64) ** 2).T)
    return np.max(np.abs(got - ref) / np.maximum(scale, 1e-30))


@pytest.mark.parametrize("t,rows,cols,seq", [
    (Q4_K, 128, 256, 512), (Q6_K, 130, 256, 513), (Q4_K, 385, 512, 608), (Q6_K, 300, 1280, 1025), (Q4_K, 1, 768, 545), (Q6_K, 200, 2048, 512),
    (Q4_K, 20000, 256, 512), (Q6_K, 19001, 512, 530), (Q4_K, 700, 2304, 4097), (Q6_K, 2100, 512, 3000), (Q6_K, 2500, 2048, 2050),
])
def test_long_prompt_matmul(ops, t, rows, cols, seq):
    rng = np.random.default_rng(rows + 7 * cols + seq)
    w, x = weights(rng, t, rows, cols), rng.standard_normal((seq, cols)).astype(np.float32)
    fn = ops.q4k_bf16_gemm_batch if t == Q4_K else ops.q6k_bf16_gemm_batch
    got = fn(w, rows, cols, x).reshape(seq, rows)
    assert off(got, t, w, rows, cols, x) <= 1e-4
    assert np.array_equal(got, fn(w, rows, cols, x).reshape(seq, rows))


@pytest.mark.parametrize("cols,seq", [(1024, 512), (1024, 700), (2048, 600)])
def test_long_prompt_matrices_of_both_formats(ops, cols, seq):
    """The two CTAs of a pair take row tiles of different matrices, and of different formats."""
    import torch

    import runnburn_b200 as r
    rng = np.random.default_rng(seq)
    types, rows = (Q4_K, Q6_K, Q4_K), (300, 129, 250)
    ws = [quantized(rng, t, n, cols)[1] for t, n in zip(types, rows)]
    x = rng.standard_normal((seq, cols)).astype(np.float32)
    wt, xt = [torch.from_numpy(np.ascontiguousarray(w)).cuda() for w in ws], torch.from_numpy(x).cuda()
    xb = torch.empty(seq * cols, dtype=torch.int16, device="cuda")
    ys = [torch.full((seq, n), float("nan"), device="cuda") for n in rows]
    assert r.load().rnb_b200_dev_prefill_gemm_multi(
        3, (ctypes.c_int * 3)(*types), (ctypes.c_void_p * 3)(*[w.data_ptr() for w in wt]), (ctypes.c_size_t * 3)(*rows),
        (ctypes.c_void_p * 3)(*[y.data_ptr() for y in ys]), cols, xt.data_ptr(), seq, xb.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert ops.dev_error_flag() == 0
    for t, n, w, y in zip(types, rows, ws, ys):
        assert off(y.cpu().numpy(), t, w, n, cols, x) <= 1e-4


@pytest.mark.parametrize("t,rows,cols,seq", [(Q4_K, 64, 1024, 257), (Q6_K, 65, 768, 300), (Q6_K, 100, 2048, 300), (Q4_K, 1000, 2048, 577), (Q4_K, 9601, 256, 320),
                                             (Q6_K, 2500, 512, 2049)])
def test_long_prompt_gate_up(ops, t, rows, cols, seq):
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


@pytest.mark.parametrize("t,rows,cols,seq", [(Q4_K, 512, 14336, 512), (Q6_K, 512, 14336, 1000), (Q4_K, 20000, 1024, 600)])
def test_long_prompt_matmul_repeats_its_bits(ops, t, rows, cols, seq):
    """Weight tiles of one CTA are read by MMAs that the other issues: 200 launches that give the same bits as the first,
    many stages deep and over several tiles per pair, the weights being the same and the tokens different from launch to
    launch, so that a stale tile would show."""
    import torch

    import runnburn_b200 as r
    rng = np.random.default_rng(cols + seq)
    w = torch.from_numpy(random_blocks(rng, t, rows, cols)).cuda()
    xs = [torch.randn(seq, cols, device="cuda", generator=torch.Generator("cuda").manual_seed(i)) for i in range(2)]
    xb = torch.empty(seq * cols, dtype=torch.int16, device="cuda")
    ys = [torch.empty(seq, rows, device="cuda") for _ in range(2)]
    want = []
    for i in range(200):
        x, y = xs[i & 1], ys[i & 1]
        assert r.load().rnb_b200_dev_prefill_gemm_multi(
            1, (ctypes.c_int * 1)(t), (ctypes.c_void_p * 1)(w.data_ptr()), (ctypes.c_size_t * 1)(rows), (ctypes.c_void_p * 1)(y.data_ptr()), cols, x.data_ptr(), seq,
            xb.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        if i < 2:
            want.append(y.clone())
        else:
            assert torch.equal(y, want[i & 1]), i
    torch.cuda.synchronize()
    assert ops.dev_error_flag() == 0
