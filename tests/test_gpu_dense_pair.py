"""The bf16 matmul of long prompts on pairs of SMs, by way of stacks whose launches have more tiles than the chip has pairs: one, three and
five stages of K (fewer than the ring has, and more), matrices of several row counts in one launch, ragged rows and tokens, f32, bf16,
decay and gate + up results; and portions of a prompt on either side of the end of the key ring.  Against the plain reference in f64; every
projection rounds its input to bf16, the bound of the stack tests (3e-2 of the rows' scale)."""
import pytest

import stack_util as su
from hybrid_ref import Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,n", [(64, 2003), (192, 1100), (320, 2048)])
@pytest.mark.parametrize("design", ["wkv", "retention", "gla", "parallel"])
def test_pairs_take_several_tiles_in_turn(design, width, n):
    # gate + up of 5000 rows: 40 tiles of rows x 3 to 5 of tokens; four projections of 1280 or 1216 rows: 20 x 3 to 5
    if design == "wkv":
        cfg = su.config([su.wkv(heads=20, dim=64, ff=5000)], width=width)
    elif design == "retention":
        cfg = su.config([su.retention(heads=19, dim=64, vdim=64, ff=5000)], width=width)
    elif design == "gla":
        cfg = su.dutivik([su.gla(heads=20, dim=64, vdim=64, ff=5000)], width=width)
    else:
        cfg = su.dutivik([su.parallel(su.window(heads=10, kv_heads=5, dim=128, vdim=128, size=200), su.delta(heads=20, kv_heads=10, dim=64, vdim=64), ff=5000)], width=width)
    w, toks = su.weights(cfg, seed=width, rank=16), su.tokens(cfg, n, seed=1)
    dec = su.decoder(cfg, w, "bfloat16", max_ctx=2048)
    got = dec.prefill_logits(toks, 0, list(range(n)))[0]
    dec.close()
    assert not (why := su.bad(got, Model(cfg, w).forward(toks), "bfloat16")), why


def test_prompt_attention_across_the_end_of_the_key_ring():
    """Keys and values of 128 elements, a window of 70: the ring holds 4165 positions.  The first portions run before it wraps, the last
    one behind."""
    cfg = su.dutivik([su.parallel(su.window(heads=4, kv_heads=2, dim=128, vdim=128, size=70, scale=128 ** -0.5), su.delta(heads=2, kv_heads=1, dim=32, vdim=32))], width=128)
    w, toks = su.weights(cfg, seed=3, rank=16), su.tokens(cfg, 4400, seed=1)
    dec = su.decoder(cfg, w, "bfloat16", max_ctx=8192)
    got = su.feed(dec, toks, [1500, 1500, 1100, 130, 170])
    dec.close()
    assert not (why := su.bad(got, Model(cfg, w).forward(toks), "bfloat16")), why
