"""Prefill matmul with tiles of up to 512 tokens (weights in shared memory): tiled copies of whole blocks, rows that they cannot
describe, both formats in one launch, gate + up, odd numbers of row tiles, ragged rows and tokens, several tiles in turn.  Which kernel a
launch takes is a rule on its sizes; every case here asserts that it is this one.

Bound: f32 accumulation only, 1e-4 of a dot product's scale sqrt(sum (x w)^2), as for the other prompt kernels."""
import ctypes

import numpy as np
import pytest

import oracle as orc
from synth import Q4_K, Q6_K, random_blocks
from test_gpu_prefill_gemm import bf16_round, ops  # noqa: F401
from test_gpu_prefill_pair import off

pytestmark = pytest.mark.gpu
SPLIT, PAIR, WIDE = 0, 1, 2


def plan(types, wt, rows, cols, seq, w2=None):
    import runnburn_b200 as r
    n, out = len(types), [ctypes.c_int() for _ in range(3)]
    assert r.load().rnb_b200_dev_prefill_gemm_plan(n, (ctypes.c_int * n)(*types), (ctypes.c_void_p * n)(*[w.data_ptr() for w in wt]),
                                                   w2.data_ptr() if w2 is not None else None, (ctypes.c_size_t * n)(*rows), cols, seq,
                                                   *[ctypes.byref(o) for o in out]) == 0
    return tuple(o.value for o in out)


def on_gpu(*arrays):
    import torch
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def multiply(ops, types, rows, cols, seq, seed):
    import torch

    import runnburn_b200 as r
    rng, n = np.random.default_rng(seed), len(types)
    ws = [random_blocks(rng, t, m, cols) for t, m in zip(types, rows)]
    x = rng.standard_normal((seq, cols)).astype(np.float32)
    wt, (xt,) = on_gpu(*ws), on_gpu(x)
    xb, ys = torch.empty(seq * cols, dtype=torch.int16, device="cuda"), [torch.full((seq, m), float("nan"), device="cuda") for m in rows]
    assert plan(types, wt, rows, cols, seq)[0] == WIDE
    assert r.load().rnb_b200_dev_prefill_gemm_multi(
        n, (ctypes.c_int * n)(*types), (ctypes.c_void_p * n)(*[w.data_ptr() for w in wt]), (ctypes.c_size_t * n)(*rows),
        (ctypes.c_void_p * n)(*[y.data_ptr() for y in ys]), cols, xt.data_ptr(), seq, xb.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert ops.dev_error_flag() == 0
    for t, m, w, y in zip(types, rows, ws, ys):
        assert off(y.cpu().numpy(), t, w, m, cols, x) <= 1e-4


@pytest.mark.parametrize("rows,cols,seq", [(9500, 2048, 385), (9500, 1280, 385), (28500, 1024, 385), (9472, 4096, 1024)])
def test_one_matrix(ops, rows, cols, seq):
    multiply(ops, (Q6_K,), (rows,), cols, seq, rows + cols)


@pytest.mark.parametrize("types,rows", [((Q4_K, Q4_K, Q6_K), (3968, 1000, 1100)), ((Q6_K, Q4_K, Q4_K), (4096, 1024, 1024))])
def test_matrices_of_both_formats(ops, types, rows):
    """Row tiles of the first launch: 31, 8 and 9, so that the two CTAs of a pair take different matrices and formats."""
    multiply(ops, types, rows, 2048, 1153, sum(rows))


@pytest.mark.parametrize("rows,cols,seq", [(4990, 4096, 1300)])
def test_one_matrix_of_four_bits(ops, rows, cols, seq):
    """An odd number of row tiles; the last tile of tokens holds 404 of 448."""
    multiply(ops, (Q4_K,), (rows,), cols, seq, rows)


def test_gate_and_up(ops):
    import torch

    import runnburn_b200 as r
    rng, rows, cols, seq = np.random.default_rng(1), 4610, 2048, 1000   # 73 row tiles
    ws, x = [random_blocks(rng, Q6_K, rows, cols) for _ in range(2)], (rng.standard_normal((seq, cols)) * 0.3).astype(np.float32)
    wt, (xt,) = on_gpu(*ws), on_gpu(x)
    xb, act = torch.empty(seq * cols, dtype=torch.int16, device="cuda"), torch.full((seq, rows), float("nan"), device="cuda").bfloat16()
    assert plan((Q6_K,), wt[:1], (rows,), cols, seq, wt[1])[0] == WIDE
    assert r.load().rnb_b200_dev_prefill_gemm_silu(Q6_K, wt[0].data_ptr(), wt[1].data_ptr(), rows, cols, xt.data_ptr(), seq, xb.data_ptr(), act.data_ptr(),
                                                   torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert ops.dev_error_flag() == 0
    xr = bf16_round(x).astype(np.float64)
    wd = [bf16_round(orc.dequantize_matrix(Q6_K, w, rows, cols).reshape(rows, cols)).astype(np.float64) for w in ws]
    g, u = (xr @ w.T for w in wd)
    want = g / (1 + np.exp(-g)) * u
    sg, su = (np.sqrt((xr ** 2) @ (w ** 2).T) for w in wd)
    # |d silu| <= 1.1; both products off by 1e-4 of their scale, then one rounding to bf16
    assert np.all(np.abs(act.float().cpu().numpy() - want) <= 1e-4 * (1.1 * sg * np.abs(u) + np.abs(g) * su) + 2.0 ** -8 * np.abs(want) + 1e-30)


@pytest.mark.parametrize("t,rows,cols,seq,want", [
    (Q6_K, 256, 256, 2, SPLIT), (Q6_K, 256, 768, 128, SPLIT), (Q6_K, 256, 768, 129, PAIR), (Q6_K, 256, 1024, 2, PAIR),   # rows of less than four blocks, 128 tokens
    (Q6_K, 9472, 4096, 300, PAIR),
    (Q4_K, 8192, 8192, 850, WIDE), (Q4_K, 11008, 4096, 1300, WIDE), (Q6_K, 14336, 4096, 1024, WIDE),   # where this kernel is the faster one by 6 %
    (Q4_K, 28672, 4096, 2048, PAIR), (Q6_K, 4096, 14336, 203, PAIR),
])
def test_the_kernel_of_a_launch(ops, t, rows, cols, seq, want):
    import torch
    assert plan((t,), [torch.empty(16, dtype=torch.uint8, device="cuda")], (rows,), cols, seq)[0] == want
