"""Prefill attention on tensor memory: sizes at the edges of its tiles (128 rows of query x head, 64 keys), every group of
heads, and rows whose maximum grows from tile to tile (the output in tensor memory is scaled) or falls, against f64.

Bound: queries and probabilities enter as two f16 terms (2^-21 of each product at worst) and sums are f32: a row's error
is below 2^-18 of the largest value of V for scores of a few units; a score of size s carries 2^-22 s into the exponent.
1e-4 of the largest output covers scores up to 200."""
import numpy as np
import pytest

from test_gpu_prefill_gemm import ops  # noqa: F401

pytestmark = pytest.mark.gpu


def reference(q, k, v, scale):
    seq, heads, _ = q.shape
    kv_len, kvh, _ = k.shape
    out = np.empty(q.shape)
    seen = np.arange(kv_len)[None] <= np.arange(seq)[:, None] + kv_len - seq
    for h in range(heads):
        s = np.where(seen, q[:, h].astype(np.float64) @ k[:, h * kvh // heads].astype(np.float64).T * scale, -np.inf)
        p = np.exp(s - s.max(1, keepdims=True))
        out[:, h] = (p / p.sum(1, keepdims=True)) @ v[:, h * kvh // heads].astype(np.float64)
    return out


@pytest.mark.parametrize("shape", ["flat", "growing", "falling"])
@pytest.mark.parametrize("heads,kvh,seq,kv_len", [
    (8, 8, 1, 1), (2, 2, 128, 128), (4, 2, 64, 65), (8, 2, 33, 129), (16, 2, 17, 300), (16, 1, 8, 64), (32, 1, 5, 191), (64, 1, 3, 192), (128, 1, 2, 257),
    (32, 8, 513, 1200), (4, 1, 640, 640),
])
def test_prefill_attention(ops, heads, kvh, seq, kv_len, shape):
    rng = np.random.default_rng(heads + 31 * seq + kv_len)
    q = rng.standard_normal((seq, heads, 128)).astype(np.float32)
    k = rng.standard_normal((kv_len, kvh, 128))
    if shape != "flat":
        # the keys share a direction with the queries, more of it towards one end: scores move by up to 60
        q += 1.0
        k += np.linspace(0.0, 5.0, kv_len)[:, None, None] * (1.0 if shape == "growing" else -1.0)
    k, v = k.astype(np.float16), rng.standard_normal((kv_len, kvh, 128)).astype(np.float16)
    scale = 1.0 / np.sqrt(128.0)
    got = ops.attention_prefill_flash_hd128_f16kv(q.reshape(-1), k.view(np.uint16).reshape(-1), v.view(np.uint16).reshape(-1), seq, kv_len, heads, kvh, scale)
    want = reference(q, k, v, scale)
    assert ops.dev_error_flag() == 0
    assert np.max(np.abs(np.asarray(got).reshape(want.shape) - want)) <= 1e-4 * np.max(np.abs(want))


@pytest.mark.parametrize("heads,kvh,seq,kv_len", [(8, 2, 33, 129), (32, 1, 5, 191)])
def test_prefill_attention_with_any_scale(ops, heads, kvh, seq, kv_len):
    """A scale of s with queries q and one of -s with -q are the same scores, a scale of zero is queries of zero: the same bits, and
    a mean over the visible keys."""
    rng = np.random.default_rng(seq)
    q = rng.standard_normal((seq, heads, 128)).astype(np.float32)
    k, v = (rng.standard_normal((kv_len, kvh, 128)).astype(np.float16) for _ in range(2))

    def run(q, scale):
        return np.asarray(ops.attention_prefill_flash_hd128_f16kv(q.reshape(-1), k.view(np.uint16).reshape(-1), v.view(np.uint16).reshape(-1), seq, kv_len, heads, kvh,
                                                                  scale)).reshape(seq, heads, 128)

    s = 1.0 / np.sqrt(128.0)
    assert np.array_equal(run(q, -s), run(-q, s))
    flat = run(q, 0.0)
    assert np.array_equal(flat, run(0.0 * q, 1.0))
    for got, scale in ((run(q, -s), -s), (flat, 0.0)):
        want = reference(q, k, v, scale)
        assert np.max(np.abs(got - want)) <= 1e-4 * np.max(np.abs(want))
    assert ops.dev_error_flag() == 0


@pytest.mark.parametrize("cuts", [[9], [63, 64, 65], [128, 129], [300]])
@pytest.mark.parametrize("kind", ["window", "wide window", "one group", "latent", "latent 64 + 64"])
def test_prompt_attention_of_mixed_stacks(kind, cuts):
    """Keys of 128 and 192 elements and values of 128 in bf16 stacks: portions that start anywhere, windows that reach part of
    a tile, heads that share keys; the bound of the stack tests."""
    import stack_util as su
    from hybrid_ref import Model
    if "latent" in kind:
        size = dict(dim=64, rot_dim=64) if "+" in kind else dict(dim=128, rot_dim=64)
        cfg = su.config([su.latent(heads=2, vdim=128, kv_rank=128, **size)], width=256)
    else:
        left = su.window(heads=4, kv_heads=4 if kind == "one group" else 2, dim=128, vdim=128, size=1000 if kind == "wide window" else 70, scale=128 ** -0.5)
        cfg = su.dutivik([su.parallel(left, su.delta(heads=2, kv_heads=1, dim=32, vdim=32))], width=256)
    w, toks = su.weights(cfg, seed=len(kind), rank=16), su.tokens(cfg, 333 if cuts != [9] else 45, seed=1)
    dec = su.decoder(cfg, w, "bfloat16", max_ctx=512)
    got = su.feed(dec, toks, cuts)
    dec.close()
    assert not (why := su.bad(got, Model(cfg, w).forward(toks), "bfloat16")), why
