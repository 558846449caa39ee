"""What a program does with this framework, as measurable cases: requests to a decoder (a prompt, then tokens one
by one) for every kind of model it runs, and a single operator call on host data.

A case of a decoder: `context` positions stand in the cache, a prompt of `prompt` tokens is prefilled behind them, then
`steps` tokens are decoded one at a time.  The tokens are the caller's (a sampler of its own, or a text being scored);
the logits of the last position come back.  Weights are random, in the formats that a model
file has; dense and MoE stacks hold K-quant blocks, the mixed stacks bf16.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from runnburn_b200 import Decoder, ModelConfig, ops
from runnburn_b200.stack import dutivik_config, punisun_config

Q4_K, Q6_K = 12, 14
BLOCK = {Q4_K: 144, Q6_K: 210}
VOCAB = 128256
EPS_DENSE, EPS_STACK = 1e-5, 1e-6
THETA = 5e5
WINDOW, CONV, LORA = 1024, 4, 64


def _decoder(name, kind, width, layers, context, prompt, steps, ff=0, kv_heads=0, vocab=VOCAB):
    return dict(name=name, kind=kind, width=width, layers=layers, ff=ff or {1024: 4096, 2048: 8192, 4096: 14336}.get(width, width * 2),
                kv_heads=kv_heads or max(width // 512, 1), vocab=vocab, context=context, prompt=prompt, steps=steps)


def listed():
    return [
        # one projection of one token through the operator interface, activations and result on the host: an engine that
        # hands single operators to the device makes hundreds of these calls per token
        dict(name="operator-q4k-4096x4096", kind="operator", type=Q4_K, rows=4096, cols=4096),
        # the smallest model of the benchmark: a draft model's step, where launches are everything
        _decoder("tiny-step", "dense", 512, 2, 100, 0, 1, ff=1024, kv_heads=2, vocab=2048),
        # a turn of a chat with a 1B-sized model: a short question behind a short history, then the answer
        _decoder("llama-1b-turn", "dense", 2048, 16, 300, 45, 16, kv_heads=8),
        # the headline benchmark: decoding with an 8B-sized model, 4096 positions in the cache
        _decoder("llama-8b-decode-4096", "dense", 4096, 32, 4096, 0, 4, kv_heads=8),
        # reading a document: one long prompt from position 0
        _decoder("llama-8b-prompt-2048", "dense", 4096, 32, 0, 2048, 0, kv_heads=8),
        # a retrieved passage pasted into a conversation: a few hundred tokens, an odd number, behind 1000 others
        _decoder("llama-8b-passage-203", "dense", 4096, 32, 1000, 203, 0, kv_heads=8),
        # decoding with a mixture of experts (128 experts, 8 of them per token), 8192 positions in the cache; a quarter of
        # the benchmark's layers, so that its weights load quickly
        _decoder("moe-decode-8192", "moe", 2048, 12, 8192, 0, 6, ff=768, kv_heads=4),
        # a whole request to a 1B-sized mixed stack: time mixing, retention and latent attention
        _decoder("punisun-1b-request", "punisun", 2048, 16, 0, 333, 16),
        # a long prompt of a stack of the same kind at 8B widths, four layers (one of each group)
        _decoder("punisun-8b-prompt-2048", "punisun", 4096, 4, 0, 2048, 0, vocab=32768),
        # a whole request to a 1B-sized stack of parallel layers: window attention, delta rule, gated linear attention
        _decoder("dutivik-1b-request", "dutivik", 2048, 12, 0, 150, 16),
        # a long prompt of an odd length of that design at 8B widths, one group of three layers
        _decoder("dutivik-8b-prompt-1999", "dutivik", 4096, 3, 0, 1999, 0, vocab=32768),
    ]


def _log(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["operator", "dense", "dense", "dense", "moe", "punisun", "dutivik"])
    if kind == "operator":
        return dict(kind=kind, type=rng.choice([Q4_K, Q6_K]), rows=_log(rng, 64, 16384), cols=256 * _log(rng, 4, 56))
    width = 2048 if kind == "moe" else rng.choice([1024, 2048, 4096])
    deep = {1024: 16, 2048: 16, 4096: 24}[width] if kind == "dense" else {1024: 12, 2048: 8, 4096: 4}[width]
    layers = rng.randint(2, deep)
    vocab = rng.choice([32768, VOCAB])
    form = rng.choice(["prompt", "turn", "decode"])
    context = prompt = steps = 0
    if kind in ("dense", "moe"):
        if form != "prompt" or kind == "moe":
            context = _log(rng, 16, 8192)
        if form != "decode" and kind == "dense":
            prompt = _log(rng, 2, 2048 if form == "prompt" else 512)
    else:
        prompt = _log(rng, 2, 2048 if form == "prompt" else 512)
    if form != "prompt" or kind == "moe":
        steps = rng.randint(1, 8)
    c = _decoder("", kind, width, layers, context, prompt, steps, ff=768 if kind == "moe" else 0,
                 kv_heads=4 if kind == "moe" else rng.choice([width // 512, width // 256]), vocab=vocab)
    del c["name"]
    return c


# ---- weights -------------------------------------------------------------------------------------
def _gpu_rng(seed, stream=0):
    return torch.Generator(device="cuda").manual_seed(seed * 1009 + stream)


def _blocks(kind, n, g, sigma):
    """n random K-quant blocks on the GPU, weights of mean zero and about the deviation `sigma`."""
    b = torch.randint(0, 256, (n, BLOCK[kind]), dtype=torch.uint8, device="cuda", generator=g)
    spread = 0.75 + 0.5 * torch.rand(n, 1, device="cuda", generator=g)
    if kind == Q4_K:
        # w = d * scale * nibble - dmin * min with min = scale and dmin = 7.5 d
        s = torch.randint(20, 64, (n, 8), dtype=torch.uint8, device="cuda", generator=g)
        d = spread * (sigma / (4.61 * 43))
        b[:, 0:4] = torch.cat([d, 7.5 * d], 1).half().view(torch.uint8)
        lo, hi = s[:, :4], s[:, 4:]
        b[:, 4:8] = b[:, 8:12] = lo | ((hi >> 4) << 6)
        b[:, 12:16] = (hi & 15) | ((hi & 15) << 4)
    else:
        s = torch.randint(40, 128, (n, 16), dtype=torch.int16, device="cuda", generator=g)
        sign = torch.randint(0, 2, (n, 16), dtype=torch.int16, device="cuda", generator=g) * 2 - 1
        b[:, 192:208] = (s * sign).to(torch.int8).view(torch.uint8)
        b[:, 208:210] = (spread * (sigma / (18.5 * 88))).half().view(torch.uint8)
    return b


def _values(kind, b):
    """The values of K-quant blocks in 64 bits, [n, 256]."""
    n = b.shape[0]
    if kind == Q4_K:
        d, dmin = b[:, 0:4].contiguous().view(torch.float16).double().unbind(1)
        s = b[:, 4:16].to(torch.int16)
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | (s[:, 0:4] >> 6 << 4)], 1)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | (s[:, 4:8] >> 6 << 4)], 1)
        q = b[:, 16:].view(n, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).double().view(n, 8, 32)
        return (q * (d[:, None] * sc)[:, :, None] - (dmin[:, None] * mn)[:, :, None]).view(n, 256)
    d = b[:, 208:210].contiguous().view(torch.float16).double()
    sc = b[:, 192:208].contiguous().view(torch.int8).double() * d
    ql, qh = b[:, :128].view(n, 2, 2, 32), b[:, 128:192].view(n, 2, 1, 32)
    lo = torch.cat([ql & 15, ql >> 4], 2)
    hi = torch.cat([(qh >> (2 * i)) & 3 for i in range(4)], 2)
    q = (lo | (hi << 4)).double() - 32
    return (q.view(n, 16, 16) * sc[:, :, None]).view(n, 256)


class _Quantised:
    """Weights of a dense or MoE stack: every matrix is a run of blocks out of one pool per type, at a place of its own."""

    def __init__(self, case, seed, host):
        self.c, D, V = case, case["width"], case["vocab"]
        self.heads = 32 if case["kind"] == "moe" else max(D // 128, 1)
        qd, kd, ff = self.heads * 128, case["kv_heads"] * 128, case["ff"]
        self.moe = case["kind"] == "moe"
        att = Q6_K if self.moe else Q4_K
        # (type, rows, columns) of a layer's matrices; attn_v, ffn_down and the LM head in Q6_K, as Q4_K_M files have them
        self.shapes = {"wq": (att, qd, D), "wk": (att, kd, D), "wv": (Q6_K, kd, D), "wo": (att, D, qd)}
        if self.moe:
            self.shapes |= {"gate_exps": (Q4_K, 128 * ff, D), "up_exps": (Q4_K, 128 * ff, D), "down_exps": (Q4_K, 128 * D, ff)}
        else:
            self.shapes |= {"gate": (Q4_K, ff, D), "up": (Q4_K, ff, D), "down": (Q6_K, D, ff)}
        self.globals = {"token_embd": (Q4_K, V, D), "output": (Q6_K, V, D)}
        # as in a trained model a layer adds little to the residual, and few experts hold most of a token's weight
        g, self.pool = _gpu_rng(seed), {}
        for t in (Q4_K, Q6_K):
            most = max(r * k // 256 for n, (u, r, k) in (self.shapes | self.globals).items() if u == t and n != "token_embd")
            self.pool[t] = _blocks(t, most + 65536, g, 0.45 / D ** 0.5)
        self.pool["token_embd"] = _blocks(Q4_K, V * D // 256, g, 1.0)
        if host:
            self.pool = {t: b.cpu().numpy() for t, b in self.pool.items()}
        self.at = np.random.default_rng(seed).integers(0, 65536, (case["layers"], 16))
        self.norm = torch.rand((2 * case["layers"] + 1, D), generator=torch.Generator().manual_seed(seed)).numpy() * 0.5 + 0.75
        self.router = [torch.randn((128, D), generator=_gpu_rng(seed, 1 + i), device="cuda") * (4.0 / D ** 0.5) for i in range(case["layers"])] if self.moe else None

    def blocks(self, layer, name):
        t, rows, cols = self.shapes[name] if layer is not None else self.globals[name]
        at = self.at[layer, list(self.shapes).index(name)] if layer is not None else 0
        return t, self.pool[name if name == "token_embd" else t][at:at + rows * cols // 256]

    def matrix(self, layer, name, rows=None):
        """Values of a matrix, or of its rows of the slice `rows`."""
        t, b = self.blocks(layer, name)
        _, n, cols = self.shapes[name] if layer is not None else self.globals[name]
        b = b.view(n, cols // 256, BLOCK[t])
        b = b if rows is None else b[rows]
        return _values(t, b.reshape(-1, BLOCK[t])).view(-1, cols)

    def description(self):
        layers = []
        for i in range(self.c["layers"]):
            ly = {n: (t, b.reshape(-1)) for n in self.shapes for t, b in [self.blocks(i, n)]}
            ly |= dict(attn_norm=self.norm[2 * i], ffn_norm=self.norm[2 * i + 1])
            if self.moe:
                ly["router"] = self.router[i].cpu().numpy()
            layers.append(ly)
        return dict(layers=layers, out_norm=self.norm[-1], **{n: (t, b.reshape(-1)) for n in self.globals for t, b in [self.blocks(None, n)]})


def _stack_config(c):
    """config.json of a mixed stack: groups of layers as the benchmark has them."""
    D, h64, h128 = c["width"], c["width"] // 64, c["width"] // 128
    mlp = {"kind": "dense", "ff": c["ff"]}
    if c["kind"] == "punisun":
        wkv = dict(type="wkv", mixer=dict(heads=h64, dim=64), mlp=mlp)
        ret = dict(type="retention", mlp=mlp, mixer=dict(heads=h128, dim=128, vdim=128, rot=dict(dims=128, base=1e4),
                                                         decay=[1.0 - 2.0 ** (-5.0 - 7.0 * i / max(h128 - 1, 1)) for i in range(h128)]))
        lat = dict(type="latent_attention", mlp=mlp,
                   mixer=dict(heads=h128, dim=128, vdim=128, rot_dim=64, kv_rank=512, scale=192 ** -0.5,
                              rot=dict(dims=64, base=1e5, scaling=dict(factor=4.0, original=2048.0, fast=24.0, slow=1.5))))
        return dict(architecture="Punisun", width=D, vocab=c["vocab"], norm=dict(eps=EPS_STACK), residual_mult=0.5,
                    loop=dict(start=0, stop=2, times=2) if c["layers"] > 4 else None, layers=[(wkv, ret, wkv, lat)[i % 4] for i in range(c["layers"])])
    par = dict(type="parallel", mlp=mlp, mixer=dict(
        left=dict(heads=h128, kv_heads=max(h128 // 4, 1), dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=WINDOW),
                  rot=dict(dims=128, base=2e5, scaling=dict(factor=4.0))),
        right=dict(heads=h128, kv_heads=max(h128 // 2, 1), dim=128, vdim=128, conv=CONV), left_scale=0.7, right_scale=0.9))
    gla = dict(type="gla", mlp=mlp, mixer=dict(heads=h128, dim=64, vdim=128, tau=12.0))
    return dict(architecture="Dutivik", width=D, vocab=c["vocab"], norm=dict(eps=EPS_STACK), embedding=dict(scale=8.0),
                layers=[dict(gla) if i % 3 == 2 else dict(par) for i in range(c["layers"])])


def _stack_weights(c, cfg, seed):
    """Name -> bf16 tensor on the GPU, of a mixed stack."""
    g, D, w = _gpu_rng(seed), c["width"], {}

    def mat(name, rows, cols, gain=1.0):
        w[name] = (torch.randn(rows, cols, device="cuda", generator=g) * (gain / cols ** 0.5)).bfloat16()

    def vec(name, n, mean=0.0, sigma=0.2):
        w[name] = (mean + sigma * torch.randn(n, device="cuda", generator=g)).bfloat16()

    w["embed"] = (torch.randn(c["vocab"], D, device="cuda", generator=g) * (0.125 if c["kind"] == "dutivik" else 1.0)).bfloat16()
    for i, ly in enumerate(cfg["layers"]):
        p, x, m = f"l{i}.", f"l{i}.mix.", ly["mixer"]
        if ly["type"] in ("gla", "parallel"):
            vec(p + "norm1", D, 1.0), vec(p + "norm1.b", D)
        else:
            vec(p + "norm1", D), vec(p + "norm1b", D), vec(p + "norm2", D), vec(p + "norm2b", D)
        if ly["type"] == "parallel":
            a, b, y, z = m["left"], m["right"], x + "left.", x + "right."
            H, G, d, V = a["heads"], a["kv_heads"], a["dim"], a["vdim"]
            mat(y + "q", H * d, D), mat(y + "k", G * d, D), mat(y + "v", G * V, D), mat(y + "g", H, D, 2.0), mat(y + "o", D, H * V)
            H, G, d, V = b["heads"], b["kv_heads"], b["dim"], b["vdim"]
            for n, rows in (("q", G * d), ("k", G * d), ("v", H * V)):
                mat(z + n, rows, D, 1.5)
                t = torch.randn(rows, CONV, device="cuda", generator=g) * 0.6
                t[:, -1] += 1.0
                w[z + n + ".conv"] = t.bfloat16()
            mat(z + "b", H, D, 2.0), mat(z + "a", H, D, 2.0), mat(z + "g", H * V, D), mat(z + "o", D, H * V)
            vec(z + "A_log", H, -1.0, 1.0), vec(z + "dt_bias", H, -1.0, 1.0), vec(z + "norm", V, 1.0)
        else:
            H, d = m["heads"], m["dim"]
            V = m.get("vdim", d)
            mat(x + "o", D, H * V)
            if ly["type"] == "wkv":
                for n in "rkvgw":
                    w[x + "mu." + n] = torch.rand(D, device="cuda", generator=g).bfloat16()
                for n in "rkvg":
                    mat(x + n, H * d, D)
                mat(x + "w1", LORA, D), mat(x + "w2", H * d, LORA), vec(x + "w0", H * d, -2.0, 1.5)
                w[x + "u"] = torch.randn(H, d, device="cuda", generator=g).bfloat16()
                vec(x + "norm", H * d, 1.0)
            elif ly["type"] == "latent_attention":
                mat(x + "q", H * (d + m["rot_dim"]), D, 2.0), mat(x + "dkv", m["kv_rank"] + m["rot_dim"], D), vec(x + "dkv.norm", m["kv_rank"], 1.0)
                mat(x + "uk", H * d, m["kv_rank"]), mat(x + "uv", H * V, m["kv_rank"])
            else:
                mat(x + "q", H * d, D), mat(x + "k", H * d, D), mat(x + "v", H * V, D), mat(x + "g", H * V, D)
                if ly["type"] == "gla":
                    mat(x + "a1", LORA, D), mat(x + "a2", H * d, LORA), vec(x + "a2.b", H * d, 1.0, 2.0), vec(x + "norm", V, 1.0)
        mat(p + "mlp.gate", c["ff"], D), mat(p + "mlp.up", c["ff"], D), mat(p + "mlp.down", D, c["ff"])
    vec("final.norm", D, 1.0 if c["kind"] == "dutivik" else 0.0)
    if c["kind"] == "dutivik":
        vec("final.norm.b", D)
    return w


# ---- the path ------------------------------------------------------------------------------------
def _tokens(c, seed):
    return np.random.default_rng(seed + 7).integers(0, c["vocab"], c["prompt"] + c["steps"])


def prepare(case, seed):
    if case["kind"] == "operator":
        ops.clear_q4k_cache()   # the weights of a program that has ended may have stood at these addresses
        w = _blocks(case["type"], case["rows"] * case["cols"] // 256, _gpu_rng(seed), 0.02).cpu().numpy().reshape(-1)
        x = np.random.default_rng(seed).standard_normal(case["cols"]).astype(np.float32)
        return dict(case=case, w=w, x=x)
    c = case
    total = c["context"] + c["prompt"] + c["steps"]
    max_ctx = max(2048, -(-total // 1024) * 1024)
    if c["kind"] in ("dense", "moe"):
        w = _Quantised(c, seed, host=True)
        moe = dict(n_expert=128, n_expert_used=8, n_ff_expert=c["ff"], n_ff=0, rope_neox=1) if w.moe else dict(n_ff=c["ff"])
        dec = Decoder(ModelConfig(n_layer=c["layers"], hidden=c["width"], n_head=w.heads, n_kv_head=c["kv_heads"], vocab=c["vocab"], max_ctx=max_ctx,
                                  rms_eps=EPS_DENSE, rope_theta=THETA, **moe))
        dec.load_description(w.description())
        dec.fill_kv_synthetic(c["context"], seed)
    else:
        cfg = _stack_config(c)
        dec = Decoder((punisun_config if c["kind"] == "punisun" else dutivik_config)(cfg, max_ctx, "bfloat16"))
        for name, t in _stack_weights(c, cfg, seed).items():
            dec.set_tensor(name, "BF16", t.reshape(-1).view(torch.uint8).cpu().numpy(), tuple(t.shape))
    return dict(case=case, decoder=dec, tokens=_tokens(c, seed))


def run(state):
    c = state["case"]
    if c["kind"] == "operator":
        return (ops.q4k_gemv if c["type"] == Q4_K else ops.q6k_gemv)(state["w"], c["rows"], c["cols"], state["x"])
    dec, tokens, pos = state["decoder"], state["tokens"], c["context"]
    if c["prompt"]:
        dec.prefill(tokens[:c["prompt"]], pos)
        pos += c["prompt"]
    for t in tokens[c["prompt"]:]:
        dec.step(t, pos)
        pos += 1
    # What a step adds to the caches and states shows in the next one's logits.  The greedy tokens stay out: where two
    # logits nearly tie, another order of a sum picks the other one.
    return {"logits": dec.read_logits()}


# ---- what it cannot do without -------------------------------------------------------------------
def _stack_sizes(c):
    """(weights of all layer runs without the LM head, bytes of state and cache read and written per token,
    operations of the mixers per token beside the matrices at the mean position of the prompt)."""
    D, h64, h128, ff, n = c["width"], c["width"] // 64, c["width"] // 128, c["ff"], c["layers"]
    mlp, mean = 3 * D * ff, c["prompt"] / 2
    if c["kind"] == "punisun":
        wkv = (5 * D * D + 2 * LORA * D + mlp, 8 * h64 * 64 * 64, 6 * h64 * 64 * 64)
        ret = (5 * D * D + mlp, 8 * h128 * 128 * 128, 6 * h128 * 128 * 128)
        lat = (h128 * 192 * D + 576 * D + 2 * D * 512 + D * D + mlp, c["prompt"] * 576 * 2, 2 * h128 * (192 + 128) * mean)
        kinds = [(wkv, ret, wkv, lat)[i % 4] for i in range(n)] + ([wkv, ret] if n > 4 else [])
    else:
        kv, kd = max(h128 // 4, 1) * 128, max(h128 // 2, 1) * 128
        att = D * (2 * D + 2 * kv + h128)
        seen = min(mean, WINDOW)
        par = (att + D * (2 * kd + 2 * D + 2 * h128) + D * D + mlp, 2 * min(c["prompt"], WINDOW) * kv * 2 + 8 * h128 * 128 * 128,
               4 * D * seen + 8 * h128 * 128 * 128)
        gla = (2 * D * h128 * 64 + 3 * D * D + LORA * (D + h128 * 64) + mlp, 8 * h128 * 64 * 128, 6 * h128 * 64 * 128)
        kinds = [gla if i % 3 == 2 else par for i in range(n)]
    return [sum(k[i] for k in kinds) for i in range(3)]


def work(case):
    c = case
    if c["kind"] == "operator":
        return {"bytes": c["rows"] * c["cols"] // 256 * BLOCK[c["type"]] + 4 * (c["rows"] + c["cols"]), "flops": 2 * c["rows"] * c["cols"]}
    D, V, L, passes = c["width"], c["vocab"], c["layers"], c["steps"] + (1 if c["prompt"] else 0)
    tokens = c["prompt"] + c["steps"]
    if c["kind"] in ("dense", "moe"):
        heads = 32 if c["kind"] == "moe" else max(D // 128, 1)
        qd, kd, ff = heads * 128, c["kv_heads"] * 128, c["ff"]
        used = 8 if c["kind"] == "moe" else 1
        att = (D * qd * 2 + D * kd) * (210 if used > 1 else 144) / 256 + D * kd * 210 / 256
        ffn = used * (2 * D * ff * 144 + D * ff * (144 if used > 1 else 210)) / 256 + (128 * D * 4 if used > 1 else 0)
        kv = 2 * kd * 2 * L
        params = L * (2 * D * qd + 2 * D * kd + 3 * used * D * ff)
        seen = c["context"] + tokens / 2
        return {"bytes": passes * (L * (att + ffn) + V * D * 210 / 256 + c["context"] * kv) + tokens * (kv + D * 144 / 256) + 4 * V,
                "flops": 2 * params * tokens + 2 * V * D * passes + 4 * L * qd * seen * tokens}
    params, state, mixers = _stack_sizes(c)
    return {"bytes": passes * (2 * params + 2 * V * D) + c["steps"] * state + tokens * D * 2 + 4 * V,
            "flops": 2 * params * tokens + 2 * V * D * passes + mixers * tokens}


def tolerance(case):
    # Activations are quantised to 8 bits (steps) or rounded to bf16 (prompts): a last-bit change in the order of a sum
    # moves some of them by one step, and later layers more.  Measured with other attention kernels (a step's in chunks
    # instead of in order, a prompt's split over the keys), another epilogue of the gate and up product, and prompts cut
    # into portions, 35 cases: 1.24e-2 with steps, 6e-3 without and for mixed stacks (largest 0.057 and 0.026); the
    # operator gave the same bits.
    if case["kind"] == "operator":
        return {"rel": 1e-5, "max": 1e-4}
    return {"rel": 0.03, "max": 0.23} if case["kind"] in ("dense", "moe") and case["steps"] else {"rel": 0.024, "max": 0.11}


# ---- the same in 64 bits -------------------------------------------------------------------------
def exact(case, seed):
    c = case
    if c["kind"] == "operator":
        w = _values(c["type"], _blocks(c["type"], c["rows"] * c["cols"] // 256, _gpu_rng(seed), 0.02)).view(c["rows"], c["cols"])
        x = np.random.default_rng(seed).standard_normal(c["cols"]).astype(np.float32)
        return w @ torch.from_numpy(x).double().cuda()
    tokens = torch.from_numpy(_tokens(c, seed)).cuda()
    return {"logits": (_exact_dense if c["kind"] in ("dense", "moe") else _exact_stack)(c, seed, tokens)}


def _mix64(z):
    def mul(a, k):
        return a * (k - (1 << 64) if k >> 63 else k)
    z = z + (0x9e3779b97f4a7c15 - (1 << 64))
    z = mul(z ^ ((z >> 30) & ((1 << 34) - 1)), 0xbf58476d1ce4e5b9)
    z = mul(z ^ ((z >> 27) & ((1 << 37) - 1)), 0x94d049bb133111eb)
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def _cache_rows(seed, n, dim):
    """The rows that a cache filled for `seed` holds: f16 normal values from a counter."""
    i = torch.arange(n * dim, device="cuda")
    r = _mix64(seed ^ (i * (0xd1342543de82ef95 - (1 << 64))))
    u1 = (((r >> 40) & 0xffffff).double() + 1) / 16777217
    u2 = (r & 0xffffff).double() / 16777216
    return (torch.sqrt(-2 * torch.log(u1)) * torch.cos(2 * math.pi * u2)).half().double().view(n, dim)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, pos0, first=0, window=None):
    """q [T, H, d] at positions pos0.., k [S, G, d], v [S, G, e] at positions first..: causal, grouped heads."""
    T, H, _ = q.shape
    S, G, e = v.shape
    out = torch.empty(T, H, e, dtype=q.dtype, device=q.device)
    at = torch.arange(S, device=q.device) + first
    for t in range(0, T, 512):
        p = torch.arange(t, min(T, t + 512), device=q.device)[:, None] + pos0
        seen = (at[None] <= p) & ((p - at[None] < window) if window else torch.ones_like(p, dtype=torch.bool))
        for h in range(H):
            s = (q[t:t + 512, h] @ k[:, h * G // H].T) * scale
            out[t:t + 512, h] = torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[:, h * G // H]
    return out


def _exact_dense(c, seed, tokens):
    w = _Quantised(c, seed, host=False)
    L, T, G = c["layers"], len(tokens), c["kv_heads"]
    norm = torch.from_numpy(w.norm).double().cuda()
    pos = torch.arange(T, device="cuda", dtype=torch.float64) + c["context"]
    angle = pos[:, None] * THETA ** (-torch.arange(0, 128, 2, device="cuda", dtype=torch.float64) / 128)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rotate(y):
        a, b = (y[..., :64], y[..., 64:]) if w.moe else (y[..., 0::2], y[..., 1::2])
        r = (a * cos - b * sin, a * sin + b * cos)
        return torch.cat(r, -1) if w.moe else torch.stack(r, -1).flatten(-2)

    x = w.matrix(None, "token_embd", tokens)
    for i in range(L):
        h = _rms(x, EPS_DENSE) * norm[2 * i]
        q, k, v = (h @ w.matrix(i, n).T for n in ("wq", "wk", "wv"))
        k = torch.cat([_cache_rows(seed * 131 + 2 * i, c["context"], G * 128).view(-1, G, 128), rotate(k.view(T, G, 128))])
        v = torch.cat([_cache_rows(seed * 131 + 2 * i + 1, c["context"], G * 128).view(-1, G, 128), v.view(T, G, 128)])
        x = x + _attend(rotate(q.view(T, -1, 128)), k, v, 128 ** -0.5, c["context"]).flatten(1) @ w.matrix(i, "wo").T
        h = _rms(x, EPS_DENSE) * norm[2 * i + 1]
        if not w.moe:
            x = x + (torch.nn.functional.silu(h @ w.matrix(i, "gate").T) * (h @ w.matrix(i, "up").T)) @ w.matrix(i, "down").T
            continue
        top, ids = (h @ w.router[i].double().T).topk(8, -1)
        share, y, ff, D = torch.softmax(top, -1), torch.zeros_like(x), c["ff"], c["width"]
        for t in range(T):
            for s, e in zip(share[t], ids[t].tolist()):
                a = torch.nn.functional.silu(w.matrix(i, "gate_exps", slice(e * ff, (e + 1) * ff)) @ h[t]) * (w.matrix(i, "up_exps", slice(e * ff, (e + 1) * ff)) @ h[t])
                y[t] += s * (w.matrix(i, "down_exps", slice(e * D, (e + 1) * D)) @ a)
        x = x + y
    return w.matrix(None, "output") @ (_rms(x[-1], EPS_DENSE) * norm[-1])


def _tables(rot, T):
    """cos, sin [T, dims / 2] of a rotation, linear or YaRN scaling included."""
    dims, base, sc, mult = rot["dims"], rot["base"], rot.get("scaling"), 1.0
    i = torch.arange(dims // 2, device="cuda", dtype=torch.float64)
    f = base ** (-2.0 * i / dims)
    if sc and "original" not in sc:
        f = f / sc["factor"]
    elif sc:
        lo, hi = (dims * math.log(sc["original"] / (2 * math.pi * sc[k])) / (2 * math.log(base)) for k in ("fast", "slow"))
        lo, hi = max(math.floor(lo), 0.0), min(math.ceil(hi), dims - 1.0)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f = f / sc["factor"] * ramp + f * (1 - ramp)
        mult = 0.1 * math.log(sc["factor"]) + 1.0
    a = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * f
    return a.cos()[:, None] * mult, a.sin()[:, None] * mult


def _turn(x, table, interleaved):
    cos, sin = table
    a, b = (x[..., 0::2], x[..., 1::2]) if interleaved else x.chunk(2, -1)
    r = (a * cos - b * sin, b * cos + a * sin)
    return torch.stack(r, -1).flatten(-2) if interleaved else torch.cat(r, -1)


def _recurrence(q, k, v, decay, bonus=None, beta=None):
    """S <- decay S + k v^T over the tokens, o = q S.  `bonus`: the state is read before the token is written, the token
    itself with that factor; `beta`: what the state answers to k is taken off v first."""
    T, H, d = k.shape
    S, out = torch.zeros(H, d, v.shape[2], dtype=k.dtype, device=k.device), torch.empty_like(v)
    for t in range(T):
        if bonus is not None:
            kv = k[t][:, :, None] * v[t][:, None]
            out[t] = torch.bmm(q[t][:, None], S + bonus[:, :, None] * kv)[:, 0]
            S = decay[t][:, :, None] * S + kv
            continue
        S = decay[t][:, :, None] * S
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None]
        out[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return out


def _exact_mixer(kind, m, w, p, h, eps):
    T, silu = h.shape[0], torch.nn.functional.silu

    def heads(x, n):
        return x.view(T, n, -1)

    def mul(x, name):
        return x @ w[p + name].double().T

    if kind == "parallel":
        a, b = m["left"], m["right"]
        left = _exact_mixer("attention", a, w, p + "left.", h, eps)
        return m["left_scale"] * left + m["right_scale"] * _exact_mixer("delta", b, w, p + "right.", h, eps)
    H, d = m["heads"], m["dim"]
    if kind == "attention":
        G, table = m["kv_heads"], _tables(m["rot"], T)
        q, k = (_rms(_turn(heads(mul(h, n), g), table, True), eps) for n, g in (("q", H), ("k", G)))
        o = _attend(q, k, heads(mul(h, "v"), G), m["scale"], 0, window=m["mask"]["size"]) * torch.sigmoid(mul(h, "g"))[:, :, None]
    elif kind == "delta":
        G, x = m["kv_heads"], {}
        for n in "qkv":
            z = mul(h, n)
            z, taps = torch.cat([z.new_zeros(CONV - 1, z.shape[1]), z]), w[p + n + ".conv"].double()
            x[n] = silu(sum(taps[:, j] * z[j:j + T] for j in range(CONV)))
        q, k = (heads(x[n], G) * torch.rsqrt((heads(x[n], G) ** 2).sum(-1, keepdim=True) + 1e-6) for n in "qk")
        rep = torch.arange(H, device="cuda") * G // H
        g = torch.exp(-w[p + "A_log"].double().exp() * torch.nn.functional.softplus(mul(h, "a") + w[p + "dt_bias"].double(), threshold=50))
        o = _recurrence(q[:, rep] * d ** -0.5, k[:, rep], heads(x["v"], H), g[:, :, None].expand(T, H, d), beta=torch.sigmoid(mul(h, "b")))
        o = _rms(o, eps) * w[p + "norm"].double() * silu(heads(mul(h, "g"), H))
    elif kind == "gla":
        z = (h @ w[p + "a1"].double().T) @ w[p + "a2"].double().T + w[p + "a2.b"].double()
        alpha = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"])
        o = _recurrence(heads(mul(h, "q"), H) * d ** -0.5, heads(mul(h, "k"), H), heads(mul(h, "v"), H), heads(alpha, H))
        o = _rms(o, eps) * w[p + "norm"].double() * silu(heads(mul(h, "g"), H))
    elif kind == "retention":
        table = _tables(m["rot"], T)
        q, k = (_turn(heads(mul(h, n), H), table, False) for n in "qk")
        decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[None, :, None].expand(T, H, d)
        o = _rms(_recurrence(q, k * d ** -0.5, heads(mul(h, "v"), H), decay), eps) * silu(heads(mul(h, "g"), H))
    elif kind == "wkv":
        last = torch.cat([h.new_zeros(1, h.shape[1]), h[:-1]])
        x = {n: h + (last - h) * w[p + "mu." + n].double() for n in "rkvgw"}
        decay = torch.exp(-torch.exp(torch.tanh(mul(x["w"], "w1")) @ w[p + "w2"].double().T + w[p + "w0"].double()))
        o = _recurrence(*(heads(mul(x[n], n), H) for n in "rkv"), heads(decay, H), bonus=w[p + "u"].double())
        o = _rms(o, eps) * w[p + "norm"].double().view(H, d) * silu(heads(mul(x["g"], "g"), H))
    else:
        table, C, e = _tables(m["rot"], T), m["kv_rank"], m["vdim"]
        q, y = heads(mul(h, "q"), H), mul(h, "dkv")
        lat = _rms(y[:, :C], eps) * w[p + "dkv.norm"].double()
        kr = _turn(y[:, None, C:], table, True).expand(T, H, -1)
        k = torch.cat([heads(lat @ w[p + "uk"].double().T, H), kr], -1)
        o = _attend(torch.cat([q[..., :d], _turn(q[..., d:], table, True)], -1), k, (lat @ w[p + "uv"].double().T).view(T, H, e), m["scale"], 0)
    return o.reshape(T, -1) @ w[p + "o"].double().T


def _exact_stack(c, seed, tokens):
    cfg = _stack_config(c)
    w, eps = _stack_weights(c, cfg, seed), EPS_STACK

    def feed_forward(p, h, act):
        return (act(h @ w[p + "gate"].double().T) * (h @ w[p + "up"].double().T)) @ w[p + "down"].double().T

    if c["kind"] == "dutivik":
        def norm(x, name):
            return torch.nn.functional.layer_norm(x, x.shape[-1:], w[name].double(), w[name + ".b"].double(), eps)
        x = w["embed"][tokens].double() * cfg["embedding"]["scale"]
        for i, ly in enumerate(cfg["layers"]):
            h = norm(x, f"l{i}.norm1")
            x = x + _exact_mixer(ly["type"], ly["mixer"], w, f"l{i}.mix.", h, eps) + feed_forward(f"l{i}.mlp.", h, torch.nn.functional.silu)
        return w["embed"].double() @ norm(x[-1:], "final.norm")[0]

    def norm(x, name):
        return _rms(x, eps) * (1.0 + w[name].double())
    e, mult = w["embed"][tokens].double(), cfg["residual_mult"]
    runs = [(i, False) for i in range(c["layers"])]
    if cfg["loop"]:
        runs[2:2] = [(0, True), (1, False)]
    x = e
    for i, again in runs:
        ly, p = cfg["layers"][i], f"l{i}."
        x = x + e if again else x
        x = x + mult * norm(_exact_mixer(ly["type"], ly["mixer"], w, p + "mix.", norm(x, p + "norm1"), eps), p + "norm1b")
        y = feed_forward(p + "mlp.", norm(x, p + "norm2"), lambda z: torch.nn.functional.gelu(z, approximate="tanh"))
        x = x + mult * norm(y, p + "norm2b")
    return w["embed"].double() @ norm(x[-1:], "final.norm")[0]
