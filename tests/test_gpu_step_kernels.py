"""Kernels of a decode step at the sizes where their splits end, bit for bit against the oracle: attention in position order (an
eighth of the positions per CTA, groups of 16, slabs of 512 positions; heads of a cluster on one or two KV heads) and the
matvec of rows that bulk copies cannot fetch; and the merge of up to 512 chunks of a context, within the bounds of that path."""
import numpy as np
import pytest

import oracle as orc
from synth import Q4_K, Q6_K, llama_description, random_blocks
from test_gpu_ops import bits_equal, ops  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kv_len", [1, 7, 8, 9, 15, 16, 17, 63, 65, 127, 255, 300, 496, 511, 512])
@pytest.mark.parametrize("heads,kvh", [(4, 2), (3, 3), (2, 2), (1, 1), (8, 1)])
def test_attention_in_position_order(ops, heads, kvh, kv_len):
    rng = np.random.default_rng(heads * 1000 + kv_len)
    q = (rng.standard_normal(heads * 128) * 3).astype(np.float32)
    k, v = (orc.f32_to_f16_bits(rng.standard_normal(kv_len * kvh * 128)) for _ in range(2))
    scale = 1.0 / np.sqrt(128.0)
    assert np.array_equal(ops.attention_decode_hd128(q, k, v, kv_len, heads, kvh, scale), orc.attention_decode(q, k, v, heads, kvh, 128, kv_len, scale))


def test_attention_in_position_order_past_a_slab():
    """A limit of 1100 positions: the second and third slab of values, in a decoder's step."""
    import runnburn_b200 as r
    desc = llama_description(seed=5, n_layer=1, hidden=256, n_head=2, n_kv_head=1, n_ff=512, vocab=512)
    n = 1100
    dec = r.Decoder(r.ModelConfig(max_ctx=n, **desc["cfg"]))
    dec.set_exact_attention_max(n)
    dec.load_description(desc)
    ref = orc.Model(desc, n)
    for pos, tok in enumerate(np.random.default_rng(1).integers(0, 512, n).tolist()):
        want = pos in (511, 512, 527, 1023, 1024, n - 1)
        got = dec.step(tok, pos, want_logits=want)
        ref_logits = ref.decode(tok, pos)
        if want:
            assert np.array_equal(got[1], ref_logits), pos
    dec.close()
    ref.close()


@pytest.mark.parametrize("t,blocks", [(Q6_K, n) for n in (1, 2, 3, 5, 7, 9, 11, 15, 17)] + [(Q4_K, 1), (Q4_K, 9)])
@pytest.mark.parametrize("rows", [1, 4, 5, 1027])
def test_matvec_rows_at_any_even_address(ops, t, blocks, rows):
    rng = np.random.default_rng(rows * 100 + blocks)
    cols = 256 * blocks
    w, x = random_blocks(rng, t, rows, cols), rng.standard_normal(cols).astype(np.float32)
    want = orc.gemv(t, w, x, rows, cols)
    assert bits_equal(ops.gemv(t, w, rows, cols, x), want)
    ops.clear_q4k_cache()
    for start in (1, 2, 6):
        backing = np.zeros(w.size + 64, np.uint8)
        backing[start:start + w.size] = w
        ops.prewarm_q4k_weights([backing])
        assert bits_equal(ops.gemv(t, backing[start:start + w.size], rows, cols, x), want), start
        ops.clear_q4k_cache()


@pytest.mark.parametrize("max_ctx,heads,kvh", [(40, 2, 1), (160, 4, 2), (3000, 2, 2), (16384, 4, 2), (16384, 2, 1)])
def test_chunks_of_a_context_merge(max_ctx, heads, kvh):
    """2, 5, 94, 296 and 512 chunks, most of them empty or ragged: more than a warp has on the way ahead, more than the threads.
    Bounds: those of the decoder's tests for this path."""
    import runnburn_b200 as r
    from synth import max_err_vs_norm
    from test_gpu_decoder import LOGIT_TOL
    desc = llama_description(seed=heads, n_layer=1, hidden=256, n_head=heads, n_kv_head=kvh, n_ff=512, vocab=512)
    dec = r.Decoder(r.ModelConfig(max_ctx=max_ctx, **desc["cfg"]))
    dec.set_exact_attention_max(0)
    dec.load_description(desc)
    ref = orc.Model(desc, 160)
    for pos, tok in enumerate(np.random.default_rng(2).integers(0, 512, min(max_ctx, 150)).tolist()):
        got = dec.step(tok, pos, want_logits=True)[1]
        assert max_err_vs_norm(got, ref.decode(tok, pos)) <= LOGIT_TOL, pos
    dec.close()
    ref.close()


def test_steps_repeat_their_bits():
    """Token and position of a step are in place before any launch of it starts: 300 steps of a latent attention layer with a key
    that dominates, ten times over on one decoder, bit for bit (a layer that read the position too early left out the
    newest key in about one step of a thousand)."""
    import stack_util as su
    cfg = su.config([su.latent(heads=2, dim=16, vdim=16, rot_dim=4, kv_rank=32, base=1e6, ff=0)], width=64, vocab=32, residual_mult=1.0)
    dec = su.decoder(cfg, su.weights(cfg, 11), "float32")
    toks = np.random.default_rng(0).integers(0, 32, 230)
    first = su.feed(dec, toks, [200] + [1] * 30)
    for _ in range(10):
        assert np.array_equal(su.feed(dec, toks, [200] + [1] * 30), first)
    dec.close()


def _step_models():
    import runnburn_b200 as r
    import stack_util as su
    from synth import moe_description

    def dense(exact, describe=llama_description):
        desc = describe(seed=3)
        dec = r.Decoder(r.ModelConfig(max_ctx=256, **desc["cfg"]))
        dec.set_exact_attention_max(256 if exact else 0)
        dec.load_description(desc)
        return dec

    def stack(cfg):
        return su.decoder(cfg, su.weights(cfg, 5), "float32")

    mixed = su.config([su.wkv(), su.retention(), su.latent()], residual_mult=1.0)
    return {"exact": lambda: dense(True), "flash": lambda: dense(False), "experts": lambda: dense(False, moe_description),
            "punisun": lambda: stack(mixed), "dutivik": lambda: stack(su.dutivik([su.parallel(), su.gla()]))}


@pytest.mark.parametrize("model", ["exact", "flash", "experts", "punisun", "dutivik"])
def test_chained_steps_repeat_the_bits_of_host_steps(model):
    """60 steps with one launch starting behind the other, fifteen times over: the logits at the end are those of steps that the host
    waits for, bit for bit, for every kind of layer (no launch reads what the one before has yet to write)."""
    dec = _step_models()[model]()
    prompt, steps = np.random.default_rng(4).integers(0, 90, 20).tolist(), 60
    token = dec.prefill(prompt, 0)
    for pos in range(20, 20 + steps):
        token, logits = dec.step(token, pos, want_logits=True)
    for _ in range(15):
        dec.prefill(prompt, 0)
        dec.step_dev(20, True)
        for _ in range(steps - 1):
            dec.step_dev(-1, True)
        dec.sync()
        assert np.array_equal(dec.read_logits(), logits)
    dec.close()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width", [124, 2044, 2048, 4092, 4096, 4097, 4100])
def test_norms_of_one_token(width, dtype):
    """Steps at the widths where the norm of one token ends (4096, multiples of 4, whole warps): root-mean-square norms with token shift
    and an embedding that is added again, and layer norms with a bias; against the plain reference, bounds of the stacks' tests."""
    import hybrid_ref as ref
    import stack_util as su
    for cfg in (su.config([su.wkv(heads=2, ff=0), su.retention(heads=1)], width=width, vocab=31, loop={"start": 0, "stop": 2, "times": 2}),
                su.dutivik([su.gla(heads=2), su.parallel(ff=0)], width=width, vocab=31)):
        w = su.weights(cfg, 3)
        toks = su.tokens(cfg, 12)
        dec = su.decoder(cfg, w, dtype)
        assert not su.bad(su.feed(dec, toks, [3] + [1] * 9), ref.Model(cfg, w).forward(toks), dtype)
        dec.close()


@pytest.mark.parametrize("rows", [1, 3, 5, 1021, 32764, 32767, 32768, 32769])
def test_results_up_to_and_past_the_direct_limit(ops, rows):
    """A result of 128 KB is written to the host by a kernel, a larger one by a copy; whole 16 bytes and ends of every size."""
    rng = np.random.default_rng(rows)
    w, x = random_blocks(rng, Q4_K, rows, 256), rng.standard_normal(256).astype(np.float32)
    assert bits_equal(ops.q4k_gemv(w, rows, 256, x), orc.gemv(Q4_K, w, x, rows, 256))
    ops.clear_q4k_cache()


@pytest.mark.parametrize("t", [Q4_K, Q6_K])
@pytest.mark.parametrize("seq", [1, 127, 128, 129])
def test_inputs_up_to_and_past_the_direct_limit(ops, t, seq):
    """128 tokens of 256 values are read where they are staged, 129 are copied first; and one call behind the other does not see the last one's."""
    rng = np.random.default_rng(seq)
    w = random_blocks(rng, t, 20, 256)
    fn = ops.q4k_gemv_batch if t == Q4_K else ops.q6k_gemv_batch
    for _ in range(3):
        x = rng.standard_normal((seq, 256)).astype(np.float32)
        assert bits_equal(fn(w, 20, 256, x).reshape(seq, 20), np.stack([orc.gemv(t, w, x[i], 20, 256) for i in range(seq)]))
    ops.clear_q4k_cache()
