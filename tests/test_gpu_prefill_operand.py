"""Prefill matmul with the weights in tensor memory: tiles of one part (up to 256 tokens) and of two, K cut over two to four pairs
of SMs, rows that start at any even address (less than eight of them, in a pair of matrices too), and blocks whose scale is infinite.

Bound: f32 accumulation only, 1e-4 of a dot product's scale sqrt(sum (x w)^2), as for the other prompt kernels; silu(gate) * up is
rounded to bf16 once more, half a unit in the last place (2^-8 at most), on products that are off by that bound."""
import ctypes

import numpy as np
import pytest

import oracle as orc
from synth import Q4_K, Q6_K, random_blocks
from test_gpu_prefill_gemm import bf16_round, ops  # noqa: F401
from test_gpu_prefill_pair import off, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,rows,cols,seq", [
    (Q6_K, 1, 1024, 1), (Q6_K, 7, 1280, 129), (Q6_K, 9, 1024, 130), (Q4_K, 129, 1024, 31), (Q4_K, 129, 1024, 33),     # few rows, all bits of a skew
    (Q6_K, 300, 1280, 256), (Q6_K, 300, 1280, 257), (Q4_K, 300, 1280, 353), (Q6_K, 300, 1792, 384), (Q4_K, 300, 1280, 385), (Q6_K, 130, 1536, 640),
    (Q4_K, 2000, 4096, 20), (Q6_K, 2100, 4352, 203), (Q4_K, 4096, 4096, 45), (Q6_K, 5000, 4096, 100), (Q6_K, 256, 11008, 203),   # cuts
    (Q6_K, 20000, 1024, 320), (Q4_K, 20000, 1024, 700),                                                              # several tiles in turn
    (Q6_K, 9472, 3072, 1024),                                                                                        # 512-token tiles
])
def test_weights_in_tensor_memory(ops, t, rows, cols, seq):
    rng = np.random.default_rng(rows + 3 * cols + seq)
    w, x = weights(rng, t, rows, cols), rng.standard_normal((seq, cols)).astype(np.float32)
    fn = ops.q4k_bf16_gemm_batch if t == Q4_K else ops.q6k_bf16_gemm_batch
    got = fn(w, rows, cols, x).reshape(seq, rows)
    assert off(got, t, w, rows, cols, x) <= 1e-4
    assert np.array_equal(got, fn(w, rows, cols, x).reshape(seq, rows))


@pytest.mark.parametrize("t,rows,cols,seq", [(Q4_K, 70, 1024, 45), (Q4_K, 1000, 2048, 300), (Q6_K, 70, 1280, 200), (Q6_K, 5, 1024, 384), (Q6_K, 130, 2048, 257), (Q6_K, 600, 4352, 60)])
def test_gate_and_up_in_tensor_memory(ops, t, rows, cols, seq):
    import torch

    import runnburn_b200 as r
    rng = np.random.default_rng(rows + cols + seq)
    ws, x = [weights(rng, t, rows, cols) for _ in range(2)], (rng.standard_normal((seq, cols)) * 0.3).astype(np.float32)
    wt, xt = [torch.from_numpy(np.ascontiguousarray(w)).cuda() for w in ws], torch.from_numpy(x).cuda()
    xb, act = torch.empty(seq * cols, dtype=torch.int16, device="cuda"), torch.full((seq, rows), float("nan"), device="cuda").bfloat16()
    assert r.load().rnb_b200_dev_prefill_gemm_silu(t, wt[0].data_ptr(), wt[1].data_ptr(), rows, cols, xt.data_ptr(), seq, xb.data_ptr(), act.data_ptr(),
                                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert ops.dev_error_flag() == 0
    xr = bf16_round(x).astype(np.float64)
    wd = [bf16_round(orc.dequantize_matrix(t, w, rows, cols).reshape(rows, cols)).astype(np.float64) for w in ws]
    g, u = (xr @ w.T for w in wd)
    want = g / (1 + np.exp(-g)) * u
    sg, su = (np.sqrt((xr ** 2) @ (w ** 2).T) for w in wd)
    # |d silu| <= 1.1; both products off by 1e-4 of their scale, then one rounding to bf16
    bound = 1e-4 * (1.1 * sg * np.abs(u) + np.abs(g) * su) + 2.0 ** -8 * np.abs(want) + 1e-30
    got = act.float().cpu().numpy()
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("t,cols,seq", [(Q6_K, 2048, 45), (Q6_K, 1280, 45), (Q6_K, 2048, 300), (Q4_K, 2048, 45), (Q6_K, 768, 45)])
def test_a_block_with_an_infinite_scale(ops, t, cols, seq):
    """Its elements are infinities of their signs, 0 x infinity where a quant or a sub-block scale is zero: rows of one sign give that
    infinity, rows of both and rows with a zero give NaN, and the other rows stay as they are."""
    rng = np.random.default_rng(cols + seq)
    rows, nb = 130, cols // 256
    w = random_blocks(rng, t, rows, cols).reshape(rows, nb, -1)
    x = np.abs(rng.standard_normal((seq, cols))).astype(np.float32) + 0.5
    d = slice(208, 210) if t == Q6_K else slice(0, 2)

    def block(row, scale, quant, zeros=()):
        b = w[row, 1]
        if t == Q6_K:
            q = np.full(256, quant)
            q[list(zeros)] = 32
            part, l = q.reshape(2, 4, 32), np.arange(32)
            for n in range(2):
                b[64 * n + l] = (part[n, 0] & 15) | ((part[n, 2] & 15) << 4)
                b[64 * n + 32 + l] = (part[n, 1] & 15) | ((part[n, 3] & 15) << 4)
                b[128 + 32 * n + l] = sum((part[n, i] >> 4) << (2 * i) for i in range(4))
            b[192:208] = 3
        else:
            b[4:16], b[2:4] = 0x11, 0
            b[16:] = 0x55 if not zeros else 0x50
        b[d] = np.frombuffer(np.float16(scale).tobytes(), np.uint8)

    block(3, np.inf, 40)
    block(64, -np.inf, 63)
    block(77, np.inf, 41, zeros=(5, 200))
    if t == Q6_K:
        block(129, np.inf, 7)
    fn = ops.q4k_bf16_gemm_batch if t == Q4_K else ops.q6k_bf16_gemm_batch
    got = fn(np.ascontiguousarray(w).reshape(-1), rows, cols, x).reshape(seq, rows)
    assert np.all(got[:, 3] == np.inf) and np.all(got[:, 64] == -np.inf) and np.all(np.isnan(got[:, 77]))
    if t == Q6_K:
        assert np.all(got[:, 129] == -np.inf)
    rest = [r for r in range(rows) if r not in (3, 64, 77, 129)]
    assert off(got[:, rest], t, np.ascontiguousarray(w[rest]).reshape(-1), len(rest), cols, x) <= 1e-4
