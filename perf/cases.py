"""What this framework is timed on: the calls its users make, over the sizes they make them at.

Seven kinds of call.  Two are the fixed decoders' surface (`AttentionCUDA.forward` over paged K/V, the int8 matrix products of
the INT8 MLP), four are single layers of the config-driven models (an attention layer with grouped heads, an attention layer
through a latent, a routed feed-forward, a linear-attention layer), and one is a whole serving call through `Engine.step`.
Sizes are those of the repository's benchmark and of its configurations at widths 1024 and 2048, and what lies between.

A layer case has the rows of `seqs` portions of up to `new` tokens each, on top of up to `ctx` tokens that earlier steps left in
the cache; `ragged` spreads both over the portions.  A pass runs the layer on a batch description made once per step, as every
layer of a model does."""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "pagedattention-based-transformer-decoder-inference-framework_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import llm_decoder as ld  # noqa: E402
from llm_decoder import _cabi, hybrid  # noqa: E402

TILE = 16
BF = torch.bfloat16
F = torch.float64
EPS = 1e-5
STRETCH = {"factor": 16.0, "original": 4096, "fast": 32.0, "slow": 1.0}
ROT_BASE = 500000.0


# ------------------------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # the headline call: one decoded token per sequence of a full batch, fp16 pages, 7B-class shape, 4K tokens of context
        dict(name="decode_f16_batch64", kind="paged", kv="f16", B=64, H=32, D=128, T=4096, prefill=False, ragged=False),
        # the smallest call: one sequence of a 12-head model some hundred tokens in; latency and launches are all of it
        dict(name="decode_f16_single", kind="paged", kv="f16", B=1, H=12, D=64, T=333, prefill=False, ragged=False),
        # int8 pages and requests of unequal length, as a running server holds them
        dict(name="decode_i8_ragged", kind="paged", kv="i8", B=48, H=32, D=128, T=2048, prefill=False, ragged=True),
        # the prompt pass of the fixed decoders
        dict(name="prompt_f16", kind="paged", kv="f16", B=4, H=32, D=128, T=2048, prefill=True, ragged=False),
        # the two int8 products of a decode step's MLP
        dict(name="int8_mlp", kind="int8_mlp", rows=256, hidden=4096, inter=11008),
        # an attention layer with grouped heads: the prompt step of a serving engine, and one token each of a full batch
        dict(name="attention_prompt", kind="attention", width=2048, heads=16, kv_heads=4, dim=128, seqs=4, new=2048, ctx=0, ragged=False),
        dict(name="attention_decode", kind="attention", width=2048, heads=16, kv_heads=4, dim=128, seqs=64, new=1, ctx=2048, ragged=False),
        # a latent-attention layer: prompt portions of unequal length, some of them continuing a cached prompt; and a decode step
        dict(name="latent_prompt_ragged", kind="latent", width=2048, heads=16, dim=128, rot_dim=64, kv_rank=512, seqs=5, new=2048, ctx=1024,
             ragged=True),
        dict(name="latent_decode", kind="latent", width=2048, heads=16, dim=128, rot_dim=64, kv_rank=512, seqs=64, new=1, ctx=2048, ragged=False),
        # a routed feed-forward over the rows of a prompt step
        dict(name="experts_prompt", kind="experts", width=2048, ff=1024, experts=8, top=2, shared=2048, rows=8192),
        # a linear-attention layer over the rows of a prompt step
        dict(name="retention_prompt", kind="retention", width=2048, heads=16, dim=64, vdim=128, seqs=4, new=2048, ctx=0, ragged=False),
        # a whole serving call: prompts of unequal length in one step, then a few decode steps, then the requests end
        dict(name="serve", kind="serve", width=1024, heads=8, kv_heads=2, dim=128, lat_heads=8, lat_dim=64, rot_dim=32, kv_rank=256, ff=2816,
             seqs=8, prompt=640, steps=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "int8_mlp", "attention", "attention", "latent", "latent", "experts", "experts",
                       "retention", "serve"])
    if kind == "decode":
        H, D = rng.choice([(12, 64), (16, 64), (32, 64), (16, 128), (32, 128)])
        T = _log(rng, 17, 4096)
        return dict(kind="paged", kv=rng.choice(["f16", "f16", "i8"]), B=_log(rng, 1, 64), H=H, D=D, T=T, prefill=False,
                    ragged=rng.random() < 0.5)
    if kind == "prompt":
        H, D = rng.choice([(12, 64), (32, 64), (16, 128), (32, 128)])
        return dict(kind="paged", kv=rng.choice(["f16", "f16", "i8"]), B=rng.randint(1, 4), H=H, D=D, T=_log(rng, 100, 2048), prefill=True,
                    ragged=False)
    if kind == "int8_mlp":
        hidden, inter = rng.choice([(768, 3072), (2048, 5632), (4096, 11008)])
        return dict(kind=kind, rows=_log(rng, 1, 512), hidden=hidden, inter=inter)
    w, heads = rng.choice([(1024, 8), (2048, 16)])
    seqs = _log(rng, 1, 64)
    if rng.random() < 0.4:
        new, ctx = 1, _log(rng, 16, 2048)                       # a decode step
    else:
        new, ctx = _log(rng, 17, max(32, 8192 // seqs if seqs > 4 else 2048)), rng.choice([0, 0, _log(rng, 16, 1024)])
    if kind == "attention":
        return dict(kind=kind, width=w, heads=heads, kv_heads=rng.choice([heads // 8, heads // 4, heads // 2]), dim=rng.choice([64, 128, 128]),
                    seqs=seqs, new=new, ctx=ctx, ragged=rng.random() < 0.6)
    if kind == "latent":
        d, r, kr = (64, 32, 256) if w == 1024 else (128, 64, 512)
        return dict(kind=kind, width=w, heads=heads, dim=d, rot_dim=r, kv_rank=kr, seqs=seqs, new=new, ctx=ctx, ragged=rng.random() < 0.6)
    if kind == "experts":
        return dict(kind=kind, width=w, ff=w // 2, experts=rng.choice([4, 8, 8, 16]), top=rng.choice([1, 2, 2]),
                    shared=rng.choice([0, w]), rows=_log(rng, 1, 8192))
    if kind == "retention":
        return dict(kind=kind, width=w, heads=heads, dim=64, vdim=128, seqs=seqs, new=new, ctx=0, ragged=rng.random() < 0.6)
    seqs = rng.randint(1, 16)
    return dict(kind="serve", width=1024, heads=8, kv_heads=2, dim=128, lat_heads=8, lat_dim=64, rot_dim=32, kv_rank=256, ff=2816,
                seqs=seqs, prompt=_log(rng, 16, 5120 // seqs if seqs > 8 else 640), steps=rng.randint(2, 6))


# ------------------------------------------------------------------------------------------------------- inputs from a seed
def _gen(seed, *more):
    s = int(seed) & 0xFFFFFFFF
    for m in more:
        s = (s * 1000003 + m + 1) & 0x7FFFFFFFFFFF
    return torch.Generator(device="cuda").manual_seed(s)


def _portions(c):
    """(cached tokens, new tokens) of every sequence: a property of the case, not of the seed."""
    r = random.Random("%d %d %d" % (c["seqs"], c["new"], c["ctx"]))
    out = []
    for _ in range(c["seqs"]):
        ctx, new = c["ctx"], c["new"]
        if c["ragged"]:
            ctx = r.randint(0 if new > 1 else ctx // 8, ctx)
            new = r.randint(max(1, new // 4), new) if new > 1 else 1
        out.append((ctx, new))
    return out


def _ctx_lens(c):
    r = random.Random("%d %d %d" % (c["B"], c["H"], c["T"]))
    lens = [r.randint(max(1, c["T"] // 8), c["T"]) for _ in range(c["B"])] if c["ragged"] else [c["T"]] * c["B"]
    lens[0] = c["T"]
    return lens


def _rows(c, seed, i, n):
    """The layer's input rows of sequence i, as a norm leaves them."""
    return torch.randn(n, c["width"], device="cuda", generator=_gen(seed, 7, i)).to(BF)


class _Weights:
    def __init__(self, seed):
        self.g = _gen(seed, 3)

    def mat(self, o, i, s=1.0):
        return (torch.randn(o, i, device="cuda", generator=self.g) * (s / math.sqrt(i))).to(BF)

    def vec(self, n, std=0.02, mean=0.0):
        return (torch.randn(n, device="cuda", generator=self.g) * std + mean).to(BF)

    def attention(self, W, p, c, width):
        H, G, D = c["heads"], c["kv_heads"], c["dim"]
        for n, rows in (("q", H * D), ("k", G * D), ("v", G * D)):
            W[p + n], W[p + n + ".b"] = self.mat(rows, width), self.vec(rows)
            W[p + n + ".conv"] = (torch.randn(rows, 4, device="cuda", generator=self.g) * 0.5).to(BF)
        W[p + "o"] = self.mat(width, H * D)

    def latent(self, W, p, c, width):
        H, D, r, V, kr = c["heads"], c["dim"], c["rot_dim"], c["dim"], c["kv_rank"]
        W[p + "q"], W[p + "dkv"], W[p + "dkv.norm"] = self.mat(H * (D + r), width), self.mat(kr + r, width), self.vec(kr, 0.02, 1.0)
        W[p + "uk"], W[p + "uv"], W[p + "g"], W[p + "sink"] = self.mat(H * D, kr), self.mat(H * V, kr), self.mat(H * V, width), self.vec(H, 1.0)
        W[p + "o"] = self.mat(width, H * V)


def _attention_cfg(c):
    return {"type": "attention", "mixer": {"heads": c["heads"], "kv_heads": c["kv_heads"], "dim": c["dim"], "vdim": c["dim"], "conv": 4,
                                           "rot": {"dims": c["dim"], "base": ROT_BASE, "scaling": STRETCH}, "scale": c["dim"] ** -0.5}}


def _latent_cfg(c):
    return {"type": "latent_attention", "mixer": {"heads": c["heads"], "dim": c["dim"], "rot_dim": c["rot_dim"], "vdim": c["dim"],
                                                  "kv_rank": c["kv_rank"], "rot": {"dims": c["rot_dim"], "base": ROT_BASE, "scaling": STRETCH},
                                                  "scale": (c["dim"] + c["rot_dim"]) ** -0.5}}


def _serve_model(c, seed):
    w, width = _Weights(seed), c["width"]
    a = dict(heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"])
    l = dict(heads=c["lat_heads"], dim=c["lat_dim"], rot_dim=c["rot_dim"], kv_rank=c["kv_rank"])
    ff = {"kind": "dense", "ff": c["ff"]}
    layers = [dict(_attention_cfg(a), mlp=ff), dict(_latent_cfg(l), mlp=ff)] * 2
    cfg = {"architecture": "Tiradra", "norm": {"eps": EPS}, "vocab": 32768, "width": width, "layers": layers, "logit_softcap": 30.0,
           "loop": {"start": 1, "stop": 3, "times": 1}, "embedding": {"bigram": {"buckets": 4093, "mul_prev": 8191, "mul_cur": 127}}}
    W = {"embed": torch.randn(32768, width, device="cuda", generator=w.g).to(BF), "head": w.mat(32768, width),
         "bigram": torch.randn(4094, width, device="cuda", generator=w.g).to(BF), "loop.step": w.vec(width).reshape(1, width),
         "final.norm": w.vec(width)}
    for i in range(4):
        p = "l%d." % i
        W[p + "norm1"], W[p + "norm2"] = w.vec(width), w.vec(width)
        if i % 2:
            w.latent(W, p + "mix.", l, width)
        else:
            w.attention(W, p + "mix.", a, width)
        W[p + "mlp.gate"], W[p + "mlp.up"], W[p + "mlp.down"] = w.mat(c["ff"], width), w.mat(c["ff"], width), w.mat(width, c["ff"])
    r = random.Random("%d %d" % (c["seqs"], c["prompt"]))
    lens = [r.randint(max(1, c["prompt"] // 5), c["prompt"]) for _ in range(c["seqs"])]
    t = random.Random(int(seed))
    toks = [[t.randrange(32768) for _ in range(n + c["steps"])] for n in lens]
    return cfg, W, lens, toks


def _layer_model(c, seed):
    """Config and weights of a one-layer model whose mixer (or feed-forward) is the case's layer."""
    w, width, W = _Weights(seed), c["width"], {}
    cfg = {"norm": {"eps": EPS}, "vocab": 32, "width": width}
    if c["kind"] in ("attention", "latent"):
        cfg.update(architecture="Tiradra", layers=[(_attention_cfg if c["kind"] == "attention" else _latent_cfg)(c)])
        (w.attention if c["kind"] == "attention" else w.latent)(W, "l0.mix.", c, width)
    elif c["kind"] == "retention":
        H, D, V = c["heads"], c["dim"], c["vdim"]
        cfg.update(architecture="Namudra", streams=1, layers=[{"type": "retention", "mixer": {
            "heads": H, "dim": D, "vdim": V, "rot": {"dims": D, "base": 10000.0}, "decay": [1.0 - 2.0 ** -(3 + 5.0 * h / H) for h in range(H)]}}])
        for n, rows in (("q", H * D), ("k", H * D), ("v", H * V), ("g", H * V)):
            W["l0.mix." + n] = w.mat(rows, width)
        W["l0.mix.o"] = w.mat(width, H * V)
    else:
        f, E = c["ff"], c["experts"]
        mlp = {"kind": "moe", "expert": {"ff": f}, "router": {"experts": E, "top": c["top"]}}
        if c["shared"]:
            mlp["shared"] = {"ff": c["shared"]}
        cfg.update(architecture="Dubarax", layers=[{"type": "attention", "mlp": mlp, "mixer": {
            "heads": 1, "kv_heads": 1, "dim": 16, "vdim": 16, "mask": {"size": 16}, "bias_max": 16, "softcap": 20.0, "scale": 0.25}}])
        for n in "qkv":
            W["l0.mix." + n], W["l0.mix." + n + ".b"] = w.mat(16, width), w.vec(16)
        W["l0.mix.o"], W["l0.mix.o.b"], W["l0.mix.rel"] = w.mat(width, 16), w.vec(width), w.vec(8).reshape(8, 1)
        for nm, ff in [("e%d." % e, f) for e in range(E)] + ([("shared.", c["shared"])] if c["shared"] else []):
            W["l0.mlp.%sgate" % nm], W["l0.mlp.%sup" % nm], W["l0.mlp.%sdown" % nm] = w.mat(ff, width), w.mat(ff, width), w.mat(width, ff)
        W["l0.mlp.router"] = w.mat(E, width)
    W.update({"embed": w.mat(32, width), "head": w.mat(32, width), "final.norm": w.vec(width), "l0.norm1": w.vec(width), "l0.norm2": w.vec(width)})
    if c["kind"] == "retention":
        W.update({"l0.hc1.in": w.vec(1, 0.0, 1.0), "l0.hc1.out": w.vec(1, 0.0, 1.0), "l0.hc1.mix": w.vec(1, 0.0, 1.0).reshape(1, 1)})
    if cfg["architecture"] == "Tiradra":
        W["bigram"] = w.mat(5, width)
        cfg["embedding"] = {"bigram": {"buckets": 4, "mul_prev": 3, "mul_cur": 1}}
    return cfg, W


def _pools(c, seed):
    """Page pools, the table and the queries of a paged case."""
    B, H, D, T = c["B"], c["H"], c["D"], c["T"]
    g = _gen(seed, 11)
    nt = -(-T // TILE)
    P = B * H * nt
    table = torch.randperm(P, generator=g, device="cuda").to(torch.int32).reshape(B, H, nt)
    if c["kv"] == "f16":
        k = torch.empty((P, TILE, D), dtype=torch.float16, device="cuda").normal_(generator=g)
        v = torch.empty((P, TILE, D), dtype=torch.float16, device="cuda").normal_(generator=g)
        ks = vs = None
    else:
        k = torch.randint(-127, 128, (P, TILE, D), dtype=torch.int8, device="cuda", generator=g)
        v = torch.randint(-127, 128, (P, TILE, D), dtype=torch.int8, device="cuda", generator=g)
        ks = torch.rand((P, TILE), device="cuda", generator=g) * 30 + 50
        vs = torch.rand((P, TILE), device="cuda", generator=g) * 30 + 50
    shape = (B, H, T, D) if c["prefill"] else (B, H, D)
    return table, k, v, ks, vs, torch.randn(shape, device="cuda", generator=g)


def _int8(c, seed):
    g = _gen(seed, 13)
    i8 = lambda *s: torch.randint(-127, 128, s, dtype=torch.int8, device="cuda", generator=g)  # noqa: E731
    vec = lambda n: torch.randn(n, device="cuda", generator=g) * 5.0  # noqa: E731
    return i8(1, c["rows"], c["hidden"]), i8(1, c["hidden"], c["inter"]), i8(1, c["inter"], c["hidden"]), vec(c["inter"]), vec(c["hidden"])


# ---------------------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    c = case
    if c["kind"] == "paged":
        table, k, v, ks, vs, q = _pools(c, seed)
        cache = ld.KVTileCache(c["kv"], device="cuda")
        cache.adopt_buffers(k, v, ks, vs)
        cache.configure_table(c["B"], c["H"], table.shape[2])
        cache.page_table_.load_host_table(table.cpu().numpy())
        lens = torch.tensor(_ctx_lens(c), dtype=torch.int32, device="cuda") if c["ragged"] else None
        return dict(c=c, cache=cache, q=q, out=torch.empty_like(q), lens=lens, temp=float(np.sqrt(c["D"])))
    if c["kind"] == "int8_mlp":
        x, w1, w2, b1, b2 = _int8(c, seed)
        return dict(c=c, x=x, w1=w1, w2=w2, b1=b1, b2=b2, h=torch.empty((1, c["rows"], c["inter"]), dtype=torch.int8, device="cuda"),
                    y=torch.empty((1, c["rows"], c["hidden"]), dtype=torch.int8, device="cuda"))
    if c["kind"] == "serve":
        cfg, W, lens, toks = _serve_model(c, seed)
        cap = sum(-(-(n + c["steps"]) // TILE) * TILE for n in lens)
        model = ld.HybridDecoder(cfg, W, "bfloat16", max_tokens=cap, max_seqs=c["seqs"], tile_size=TILE)
        return dict(c=c, engine=ld.Engine(model), lens=lens, toks=toks)
    cfg, W = _layer_model(c, seed)
    portions = _portions(c) if c["kind"] != "experts" else [(0, 1)]
    cap = sum(-(-(a + b) // TILE) * TILE for a, b in portions)
    model = ld.HybridDecoder(cfg, W, "bfloat16", max_tokens=cap, max_seqs=len(portions), tile_size=TILE)
    layer = model.layers[0]
    if c["kind"] == "experts":
        g = _gen(seed, 17)
        return dict(c=c, model=model, layer=layer, h=_rows(c, seed, 0, c["rows"]), x=torch.randn(c["rows"], c["width"], device="cuda", generator=g))
    slots = [model.states.alloc() for _ in portions]
    rows = [_rows(c, seed, i, a + b) for i, (a, b) in enumerate(portions)]
    todo, held = [], 0
    for i, (a, _b) in enumerate(portions):      # what earlier steps cached
        if a:
            todo.append(i)
            held += a
        if todo and (held >= 8192 or i + 1 == len(portions)):
            batch = model.states.make_batch([(slots[j], [0] * portions[j][0]) for j in todo])
            layer.mixer.forward(hybrid._Ctx(model, batch), torch.cat([rows[j][:portions[j][0]] for j in todo]))
            todo, held = [], 0
    batch = model.states.make_batch([(s, [0] * b) for s, (_a, b) in zip(slots, portions)])
    return dict(c=c, model=model, layer=layer, batch=batch, h=torch.cat([r[a:] for r, (a, _b) in zip(rows, portions)]))


class _Rows:
    """The batch description that a routed feed-forward needs: how many rows there are."""

    def __init__(self, rows):
        self.rows = rows


def run(state):
    s, c = state, state["c"]
    if c["kind"] == "paged":
        ld.AttentionCUDA.forward(s["q"], s["out"], c["B"], c["H"], c["D"], c["T"], None, s["cache"], None, c["prefill"], c["kv"] == "f16",
                                 True, s["temp"], ctx_lens=s["lens"])
        return s["out"]
    if c["kind"] == "int8_mlp":
        M, K, N = c["rows"], c["hidden"], c["inter"]
        if not (ld.dnnl_matmul_int8(s["x"], s["w1"], s["h"], 1, M, N, K, 1.0 / 127.0, 1.0 / 127.0, math.sqrt(K) / 120.0, s["b1"], "relu") and
                ld.dnnl_matmul_int8(s["h"], s["w2"], s["y"], 1, M, K, N, 1.0 / 127.0, 1.0 / 127.0, math.sqrt(N) / 300.0, s["b2"], "")):
            raise RuntimeError("dnnl_matmul_int8 failed")
        return s["h"], s["y"]
    if c["kind"] == "serve":
        eng, out = s["engine"], []
        out.append(eng.step([(i, t[:n], [n - 1]) for i, (t, n) in enumerate(zip(s["toks"], s["lens"]))]))
        for k in range(c["steps"]):
            out.append(eng.step([(i, [t[n + k]], [0]) for i, (t, n) in enumerate(zip(s["toks"], s["lens"]))]))
        for i in range(c["seqs"]):
            eng.finish(i)
        return out
    if c["kind"] == "experts":
        ctx = hybrid._Ctx(s["model"], _Rows(c["rows"]))
        ff = s["layer"].ff.forward(ctx, s["h"])
        out = torch.empty_like(s["h"])
        # the layer's outputs join the residual, with the norm in front of the next sublayer
        _cabi.check(_cabi.lib().pa_residual_add_prenorm(
            s["x"].data_ptr(), c["rows"], c["width"], None, 1.0, None, 1.0, _cabi.ptr(ff.get("routed")), _cabi.ptr(ff.get("sel_w")),
            ff["top"], _cabi.ptr(ff.get("shared")), None, EPS, s["layer"].gain1.data_ptr(), out.data_ptr(), 2, _cabi.stream()),
            "pa_residual_add_prenorm")
        return s["x"], out
    y = s["layer"].mixer.forward(hybrid._Ctx(s["model"], s["batch"]), s["h"])
    if c["kind"] == "retention":
        return y, s["layer"].mixer.core.state
    return y


# ------------------------------------------------------------------------------------------------------------ work, tolerance
def _pairs(c):
    return sum(b * a + b * (b + 1) // 2 for a, b in _portions(c))


def work(case):
    c = case
    if c["kind"] == "paged":
        B, H, D, T = c["B"], c["H"], c["D"], c["T"]
        e = 2 if c["kv"] == "f16" else 1
        tok = sum(_ctx_lens(c))
        kv = tok * H * (2 * D * e + (8 if e == 1 else 0))
        if c["prefill"]:
            return {"bytes": kv + 8 * B * H * T * D, "flops": 4 * B * H * D * T * (T + 1) / 2}
        return {"bytes": kv + 8 * B * H * D, "flops": 4 * tok * H * D}
    if c["kind"] == "int8_mlp":
        M, K, N = c["rows"], c["hidden"], c["inter"]
        return {"bytes": 2 * K * N + M * (2 * K + N), "flops": 4 * M * N * K}
    w = c["width"]
    if c["kind"] == "experts":
        R, pairs = c["rows"], c["rows"] * c["top"]
        used = min(c["experts"], pairs)
        wts = 3 * w * (used * c["ff"] + c["shared"])
        return {"bytes": 2 * wts + R * w * (2 + 8 + 2), "flops": 6 * w * (pairs * c["ff"] + R * c["shared"])}
    if c["kind"] == "serve":
        S = c["steps"]
        r = random.Random("%d %d" % (c["seqs"], c["prompt"]))
        lens = [r.randint(max(1, c["prompt"] // 5), c["prompt"]) for _ in range(c["seqs"])]
        att = w * (2 * c["heads"] + 2 * c["kv_heads"]) * c["dim"]
        H, D, rr, kr = c["lat_heads"], c["lat_dim"], c["rot_dim"], c["kv_rank"]
        lat = w * (H * (D + rr) + kr + rr + 2 * H * D) + 2 * H * D * kr
        wts = 2 * (att + lat) + 4 * 3 * w * c["ff"]
        head = 32768 * w
        tok = sum(lens) + S * c["seqs"]
        flops = 2 * wts * tok + 2 * head * c["seqs"] * (S + 1)
        pairs = sum((n + S) * (n + S + 1) // 2 for n in lens)
        flops += 2 * pairs * (4 * c["heads"] * c["dim"] + H * (2 * (D + rr) + 2 * D))
        return {"bytes": (S + 1) * 2 * (wts + head), "flops": flops}
    R = sum(b for _a, b in _portions(c))
    if c["kind"] == "retention":
        H, D, V = c["heads"], c["dim"], c["vdim"]
        wts = w * H * (2 * D + 3 * V)
        return {"bytes": 2 * wts + 4 * R * w + 8 * c["seqs"] * H * D * V, "flops": 2 * wts * R + 6 * R * H * D * V}
    ctx = sum(a for a, _b in _portions(c))
    H, D = c["heads"], c["dim"]
    if c["kind"] == "attention":
        G = c["kv_heads"]
        wts = w * D * (2 * H + 2 * G)
        return {"bytes": 2 * wts + 4 * R * w + 4 * (ctx + R) * G * D, "flops": 2 * wts * R + 4 * _pairs(c) * H * D}
    r, kr = c["rot_dim"], c["kv_rank"]
    wts = w * (H * (D + r) + kr + r + 2 * H * D) + 2 * H * D * kr
    # per (query, key) pair and head the cheaper of the two forms of this layer: keys and values built from the latent
    per = 2 * (D + r) + 2 * D
    return {"bytes": 2 * wts + 4 * R * w + 2 * (ctx + R) * (kr + r), "flops": 2 * wts * R + _pairs(c) * H * per}


def tolerance(case):
    c = case
    if c["kind"] == "paged":
        if c["prefill"]:
            return {"rel": 1e-3, "max": 0.04}       # fp16 operands: 2.5e-4 from the float64 result
        return {"rel": 1e-5, "max": 4e-4} if c["kv"] == "f16" else {"rel": 2e-4, "max": 8e-3}   # 2.4e-7 and 5e-5 from it
    if c["kind"] == "int8_mlp":
        return "exact"
    if c["kind"] == "serve":
        return {"rel": 1.6e-2, "max": 0.4}      # 4e-3 from the float64 result
    return {"rel": 1.6e-2, "max": 0.4}          # bfloat16 operands and results: 2e-3 to 5.6e-3


# -------------------------------------------------------------------------------------------------------------------- exact
def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _sigmoid(x):
    return 1.0 / (1.0 + torch.exp(-x))


def _frequencies(dims, stretch):
    base = ROT_BASE if stretch else 10000.0
    f = [base ** (-2.0 * i / dims) for i in range(dims // 2)]
    if not stretch:
        return torch.tensor(f, dtype=F, device="cuda"), 1.0
    turns = lambda t: dims * math.log(STRETCH["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(turns(STRETCH["fast"])), 0), min(math.ceil(turns(STRETCH["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    f = [a / STRETCH["factor"] * r + a * (1.0 - r) for a, r in zip(f, ramp)]
    return torch.tensor(f, dtype=F, device="cuda"), 0.1 * math.log(STRETCH["factor"]) + 1.0


def _turn(x, dims, stretch=True):
    """x [T, heads, dim] turned by position; neighbouring entries are a pair (stretch), or entries of the two halves."""
    f, m = _frequencies(dims, stretch)
    ang = torch.arange(x.shape[0], dtype=F, device="cuda")[:, None] * f
    cs, sn = torch.cos(ang)[:, None] * m, torch.sin(ang)[:, None] * m
    y = x.clone()
    a, b = (slice(0, dims, 2), slice(1, dims, 2)) if stretch else (slice(0, dims // 2), slice(dims // 2, dims))
    y[..., a], y[..., b] = x[..., a] * cs - x[..., b] * sn, x[..., b] * cs + x[..., a] * sn
    return y


def _attend(q, k, v, scale, sink=None):
    """The last q.shape[0] positions of a sequence attend causally; q [n, H, d], k [T, G, d], v [T, G, e]."""
    n, H = q.shape[:2]
    T, G = k.shape[:2]
    out = torch.empty(n, H, v.shape[2], dtype=F, device="cuda")
    for lo in range(0, n, 1024):
        m = min(1024, n - lo)
        hidden = torch.arange(T, device="cuda")[None] > torch.arange(T - n + lo, T - n + lo + m, device="cuda")[:, None]
        for h in range(H):
            s = (q[lo:lo + m, h] @ k[:, h * G // H].T * scale).masked_fill_(hidden, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].expand(m, 1)], 1)
            out[lo:lo + m, h] = torch.softmax(s, -1)[:, :T] @ v[:, h * G // H]
    return out


def _conv(u, w):
    y = u * w[:, -1]
    for j in range(1, w.shape[1]):
        y[j:] += u[:-j] * w[:, -1 - j]
    return y


def _attention64(h, W, p, c, n):
    T, H, G, D = h.shape[0], c["heads"], c["kv_heads"], c["dim"]
    q, k, v = (_conv(h @ W[p + x].T + W[p + x + ".b"], W[p + x + ".conv"]) for x in "qkv")
    q, k = (_rms(_turn(x.reshape(T, -1, D), D)) for x in (q, k))
    return _attend(q[T - n:], k, v.reshape(T, G, D), D ** -0.5).reshape(n, H * D) @ W[p + "o"].T


def _latent64(h, W, p, c, n):
    T, H, D, r, kr = h.shape[0], c["heads"], c["dim"], c["rot_dim"], c["kv_rank"]
    q = (h @ W[p + "q"].T).reshape(T, H, D + r)
    q = torch.cat([q[..., :D], _turn(q[..., D:], r)], -1)
    down = h @ W[p + "dkv"].T
    lat = _rms(down[:, :kr]) * W[p + "dkv.norm"]
    k = torch.cat([(lat @ W[p + "uk"].T).reshape(T, H, D), _turn(down[:, None, kr:], r).expand(T, H, r)], -1)
    o = _attend(q[T - n:], k, (lat @ W[p + "uv"].T).reshape(T, H, D), (D + r) ** -0.5, W[p + "sink"]).reshape(n, H * D)
    return (o * _sigmoid(h[T - n:] @ W[p + "g"].T)) @ W[p + "o"].T


def _retention64(h, W, p, c):
    T, H, D, V = h.shape[0], c["heads"], c["dim"], c["vdim"]
    q, k = (_turn((h @ W[p + x].T).reshape(T, H, D), D, False) for x in "qk")
    k, v = k * D ** -0.5, (h @ W[p + "v"].T).reshape(T, H, V)
    decay = torch.tensor([1.0 - 2.0 ** -(3 + 5.0 * i / H) for i in range(H)], dtype=torch.float32).to("cuda", F)
    S, out = torch.zeros(H, D, V, dtype=F, device="cuda"), torch.empty(T, H, V, dtype=F, device="cuda")
    for lo in range(0, T, 256):         # blocks of 256 tokens: what came before through S, the block's own pairs in matrix form
        n = min(256, T - lo)
        t = torch.arange(n, device="cuda", dtype=F)
        a, b, e = q[lo:lo + n].transpose(0, 1), k[lo:lo + n].transpose(0, 1), v[lo:lo + n].transpose(0, 1)
        d = (t[:, None] - t[None])
        wgt = torch.where(d >= 0, decay[:, None, None] ** d.clamp(min=0), torch.zeros((), dtype=F, device="cuda"))
        o = ((a @ b.transpose(1, 2)) * wgt) @ e + (a @ S) * decay[:, None, None] ** (t + 1)[:, None]
        out[lo:lo + n] = o.transpose(0, 1)
        S = S * decay[:, None, None] ** n + (b * decay[:, None, None] ** (n - 1 - t)[:, None]).transpose(1, 2) @ e
    o = _rms(out).reshape(T, H * V)
    g = h @ W[p + "g"].T
    return (o * g * _sigmoid(g)) @ W[p + "o"].T, S


def _paged64(c, seed):
    B, H, D, T = c["B"], c["H"], c["D"], c["T"]
    table, k, v, ks, vs, q = _pools(c, seed)
    out = torch.empty(q.shape, dtype=F, device="cuda")
    for b, n in enumerate(_ctx_lens(c)):
        for h in range(H):
            ids = table[b, h].long()
            kk, vv = k[ids].to(F), v[ids].to(F)
            if ks is not None:
                kk, vv = kk / ks[ids].to(F)[..., None], vv / vs[ids].to(F)[..., None]
            kk, vv = kk.reshape(-1, 1, D)[:n], vv.reshape(-1, 1, D)[:n]
            x = q[b, h].to(F).reshape(-1, 1, D)
            out[b, h] = _attend(x, kk, vv, D ** -0.5).reshape(out[b, h].shape)
    return out


def _experts64(c, seed):
    _cfg, W = _layer_model(c, seed)
    W = {n: t.to(F) for n, t in W.items() if n.startswith("l0.mlp.") or n == "l0.norm1"}
    h = _rows(c, seed, 0, c["rows"]).to(F)
    x = torch.randn(c["rows"], c["width"], device="cuda", generator=_gen(seed, 17)).to(F)
    expert = lambda h, n: (lambda g: (g * _sigmoid(g) * (h @ W["l0.mlp.%sup" % n].T)) @ W["l0.mlp.%sdown" % n].T)(h @ W["l0.mlp.%sgate" % n].T)  # noqa: E731
    s, ids = torch.topk(torch.softmax(h @ W["l0.mlp.router"].T, -1), c["top"])
    for e in range(c["experts"]):
        rows, place = torch.nonzero(ids == e, as_tuple=True)
        if rows.numel():
            x.index_add_(0, rows, s[rows, place][:, None] * expert(h[rows], "e%d." % e))
    if c["shared"]:
        x += expert(h, "shared.")
    return x, _rms(x) * (1.0 + W["l0.norm1"])


def _serve64(c, seed):
    _cfg, W, lens, toks = _serve_model(c, seed)
    W = {n: t.to(F) for n, t in W.items()}
    a = dict(heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"])
    l = dict(heads=c["lat_heads"], dim=c["lat_dim"], rot_dim=c["rot_dim"], kv_rank=c["kv_rank"])
    norm = lambda x, w: _rms(x) * (1.0 + w)  # noqa: E731
    out = []
    for t, n in zip(toks, lens):
        ids = torch.tensor(t, device="cuda")
        pair = torch.cat([torch.tensor([4093], device="cuda"), (ids[:-1] * 8191 + ids[1:] * 127) % 4093])
        x = W["embed"][ids] + W["bigram"][pair]
        for i in range(4):
            p = "l%d." % i
            if i == 1:
                x = x + W["loop.step"][0]
            h, f = norm(x, W[p + "norm1"]), norm(x, W[p + "norm2"])
            y = _latent64(h, W, p + "mix.", l, len(t)) if i % 2 else _attention64(h, W, p + "mix.", a, len(t))
            g = f @ W[p + "mlp.gate"].T
            g = 0.5 * g * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (g + 0.044715 * g ** 3)))
            x = x + y + (g * (f @ W[p + "mlp.up"].T)) @ W[p + "mlp.down"].T
        out.append(30.0 * torch.tanh(norm(x[n - 1:], W["final.norm"]) @ W["head"].T / 30.0))
    return [torch.stack([o[k] for o in out]) for k in range(c["steps"] + 1)]


def exact(case, seed):
    c = case
    if c["kind"] == "int8_mlp":
        return None             # whole numbers
    if c["kind"] == "paged":
        return _paged64(c, seed)
    if c["kind"] == "experts":
        return _experts64(c, seed)
    if c["kind"] == "serve":
        return _serve64(c, seed)
    _cfg, W = _layer_model(c, seed)
    W = {n: t.to(F) for n, t in W.items() if n.startswith("l0.mix.")}
    out, states = [], []
    for i, (a, b) in enumerate(_portions(c)):
        h = _rows(c, seed, i, a + b).to(F)
        if c["kind"] == "retention":
            y, S = _retention64(h, W, "l0.mix.", c)
            out.append(y)
            states.append(S)
        else:
            out.append((_attention64 if c["kind"] == "attention" else _latent64)(h, W, "l0.mix.", c, b))
    if c["kind"] == "retention":
        return torch.cat(out), torch.stack(states).reshape(len(states), -1)
    return torch.cat(out)
