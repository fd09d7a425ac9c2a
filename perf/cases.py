"""The work that programs have this engine do, as cases to time and compare.

Two kinds of case.  `serve` is a whole call: an engine of the benchmark's LFM2 shapes takes the prompts of some requests
in one step and then decodes given tokens, one `Engine.step` each, logits out.  The others are one layer's part each
(`part`), run through the part's own forward() over the paged cache for one step of the engine: a portion of the prompts
of `requests` requests (`rows` tokens in all, unequal shares), behind `history` tokens that the cache holds already, or
one token a request (`rows` == `requests`: a decode step).  A decode step's case runs `layers` such parts one after
another, each with weights and a cache of its own, as the layers of a model follow one another: their matrices then come
from memory, not from the L2.  The engine replays its steps from CUDA graphs; so does a part's case: the graph is
recorded in prepare(), as the engine records a step's once and replays it for every step of that shape.

`width`, head sizes, ranks, windows and feed-forwards are those of the benchmark's configurations of each design.
"""
from __future__ import annotations

import gc
import math

import torch
import torch.nn.functional as F

from fellm_b200 import ops
from fellm_b200.cache.manager import CacheManager
from fellm_b200.parts.base import build_part
from fellm_b200.parts.spec import PartSpec

DEV = "cuda"
PAGE = 64
EPS = 1e-5
SHAPES = {"350m": (1024, 16, 4608), "700m": (1536, 24, 7168), "1.2b": (2048, 32, 8192)}       # width, heads, feed-forward
VOCAB = 65536
LAYERS, ATTENTION_LAYERS = 16, (2, 5, 8, 10, 12, 14)


# ----------------------------------------------------------------------------------------------------------- the cases

def listed():
    return [
        # one chat turn at batch 1: a short prompt, then tokens one by one.  Latency: launches and small products.
        dict(name="chat", part="serve", shape="350m", requests=1, rows=100, tokens=24),
        # a server's batch: 16 requests with prompts of unequal lengths in one step, then decoded together.
        dict(name="serve_batch", part="serve", shape="700m", requests=16, rows=1800, tokens=8),
        # the gated feed-forward of a long prompt's portion, the largest share of a prompt's arithmetic
        dict(name="swiglu_prompt", part="swiglu", dtype="bfloat16", width=2048, requests=1, rows=2048, history=0, layers=1),
        # the 32-bit engine: LFM2's attention layer over the rest of a prompt
        dict(name="attention_float32", part="attention_lfm2", dtype="float32", width=1024, requests=2, rows=201, history=300, layers=1),
        # gated delta rule over a long prompt
        dict(name="delta_prompt", part="delta", dtype="bfloat16", width=2048, requests=1, rows=2048, history=0, layers=1),
        # chunked soft-capped attention beside time mixing, two prompts in a step
        dict(name="parallel_prompt", part="parallel", dtype="bfloat16", width=1024, requests=2, rows=1100, history=0, layers=1),
        # gated linear recurrence (the forget gate writes) over three prompts of unequal lengths
        dict(name="hgrn2_prompts", part="hgrn2", dtype="bfloat16", width=1024, requests=3, rows=1537, history=0, layers=1),
        # latent attention: a prompt's portion, and single tokens of a batch behind long contexts
        dict(name="latent_prompt", part="latent", dtype="bfloat16", width=2048, requests=1, rows=2048, history=0, layers=1),
        dict(name="latent_decode", part="latent", dtype="bfloat16", width=1024, requests=8, rows=8, history=1500, layers=6),
        # windowed attention: values that are the keys, biases by distance, over a prompt; and with an output gate, decoding
        dict(name="window_prompt", part="attention_samusun", dtype="bfloat16", width=1024, requests=1, rows=2048, history=0, layers=1),
        dict(name="window_decode", part="attention_nalizen", dtype="bfloat16", width=1024, requests=12, rows=12, history=1100, layers=6),
        # routed experts for a decode step of a small batch: every expert's matrices for a handful of rows
        dict(name="experts_decode", part="experts", dtype="bfloat16", width=1024, requests=8, rows=8, history=0, layers=2),
    ]


PARTS = ("swiglu", "attention_lfm2", "delta", "channel_delta", "parallel", "hgrn2", "latent", "attention_samusun",
         "attention_nalizen", "experts")
RECURRENT = ("delta", "channel_delta", "parallel", "hgrn2")


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.15:
        n = _log_int(rng, 1, 24)
        return dict(part="serve", shape=rng.choice(("350m", "700m")), requests=n, rows=n * _log_int(rng, 12, max(13, 1800 // n)) + rng.randrange(n),
                    tokens=rng.randint(4, 24 if n < 4 else 8))
    part = rng.choice(PARTS)
    case = dict(part=part, dtype="bfloat16", width=rng.choice((1024, 2048)), history=0)
    if rng.random() < 0.35:                      # a decode step
        case["requests"] = case["rows"] = _log_int(rng, 1, 48)
    else:                                        # portions of prompts
        case["requests"] = rng.randint(1, 4)
        case["rows"] = _log_int(rng, 3 * case["requests"], 2048)
    if part.startswith("attention") or part == "latent":
        case["history"] = rng.choice((0, _log_int(rng, 10, 3000)))
    case["layers"] = 1 if case["rows"] > case["requests"] else 2 if part == "experts" else 4
    if rng.random() < 0.1:                       # the 32-bit engine
        case["dtype"], case["width"] = "float32", 1024
        case["rows"] = case["requests"] if case["rows"] == case["requests"] else min(case["rows"], 256)
        case["history"] = min(case["history"], 500)
    return case


def shares(case):
    """Rows of every request of the step: unequal where there are more rows than requests."""
    n, R = case["requests"], case["rows"]
    if R == n:
        return [1] * n
    cuts = [R * (i * (i + n)) // (n * (2 * n)) for i in range(n)] + [R]
    got = [max(1, cuts[i + 1] - cuts[i]) for i in range(n)]
    got[-1] = R - sum(got[:-1])
    return got


def histories(case):
    """Tokens every request has in the cache before the step: from two thirds of `history` up to it."""
    n, h = case["requests"], case["history"]
    return [h - (h // 3) * i // n for i in range(n)]


# ------------------------------------------------------------------------------------------------- inputs and weights

def _gen(seed, what=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1009 + what)
    return g


def _normal(g, shape, std, dtype):
    return (torch.randn(shape, generator=g, device=DEV, dtype=torch.float32) * std).to(dtype)


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float32) * (hi - lo) + lo


SCALED = dict(factor=8.0, original=4096.0, fast=32.0, slow=1.0)
BANDS = dict(factor=8.0, low=1.0, high=4.0, original=4096.0)


def make(case):
    """(category, PartSpec, [(local name, shape, kind of values, a, b)]) of the case's part."""
    d, part = case["width"], case["part"]
    W = []                    # matrices 'm' (normal, std), vectors 'n' (normal, std) and 'u' (uniform, lo, hi)
    std = d ** -0.5

    def mat(name, rows, cols, s=None):
        W.append((name, (rows, cols), "m", cols ** -0.5 if s is None else s, 0.0))

    def vec(name, shape, kind, a, b=0.0):
        W.append((name, shape, kind, a, b))

    if part == "swiglu":
        ff = {1024: 4608, 2048: 8192}[d]
        mat("gate.weight", ff, d), mat("up.weight", ff, d), mat("down.weight", d, ff)
        return "feed_forward", PartSpec.make("swiglu", size=d, ff=ff), W
    if part == "experts":
        ff, E, ident = {1024: 3328, 2048: 6144}[d], 8, 4
        mat("router.weight", E + ident, d, 2 * std)
        vec("correction", (E + ident,), "n", 0.1)
        for e in range(E):
            mat(f"e{e}.gate.weight", ff, d), mat(f"e{e}.up.weight", ff, d), mat(f"e{e}.down.weight", d, ff)
        return "feed_forward", PartSpec.make("moe", size=d, ff=ff, experts=E, identity=ident, top=2, score="softmax",
                                             correction=True, groups=(4, 2, 1)), W
    if part == "attention_lfm2":
        H, G, hd = d // 64, (d // 64) // 2, 64
        if d == 2048:
            G = 8
        mat("q_proj.weight", H * hd, d), mat("k_proj.weight", G * hd, d), mat("v_proj.weight", G * hd, d), mat("out_proj.weight", d, H * hd)
        vec("q_norm.weight", (hd,), "u", 0.5, 1.5), vec("k_norm.weight", (hd,), "u", 0.5, 1.5)
        return "mixer", PartSpec.make("attention", size=d, heads=H, kv_heads=G, head_dim=hd, qk_norm=True, norm_eps=EPS,
                                      position=PartSpec.make("rope", rot_dim=hd, theta=1000000.0, pairing="split_half")), W
    if part == "attention_samusun":
        H, hd = d // 64, 64
        G = H // 4
        mat("q_proj.weight", H * hd, d), mat("k_proj.weight", G * hd, d), mat("out_proj.weight", d, H * hd)
        vec("q_proj.bias", (H * hd,), "n", 0.02), vec("k_proj.bias", (G * hd,), "n", 0.02), vec("out_proj.bias", (d,), "n", 0.02)
        return "mixer", PartSpec.make("attention", size=d, heads=H, kv_heads=G, head_dim=hd, qk_norm=False, norm_eps=EPS,
                                      position=PartSpec.make("none"), window=1024, scale=0.125, bias=True, values_are_keys=True,
                                      slope_exp=8.0, q_temp=(0.25, 128)), W
    if part == "attention_nalizen":
        H, hd = d // 64, 64
        G = H // 4
        mat("q_proj.weight", H * hd, d), mat("k_proj.weight", G * hd, d), mat("v_proj.weight", G * hd, d)
        mat("out_gate.weight", H * hd, d), mat("out_proj.weight", d, H * hd)
        b = BANDS
        return "mixer", PartSpec.make("attention", size=d, heads=H, kv_heads=G, head_dim=hd, v_dim=hd, qk_norm=False, unit_qk_norm=True,
                                      out_gate=True, norm_eps=EPS, window=1024, scale=0.125,
                                      position=PartSpec.make("rope", rot_dim=32, theta=10000.0, pairing="split_half", table64=True,
                                                             bands=(b["factor"], b["low"], b["high"], b["original"]))), W
    if part in ("delta", "channel_delta"):
        H, dk, dv, L, R = d // 128, 128, 128, 4, 16
        G = H // 2
        for t, n in (("q", G * dk), ("k", G * dk), ("v", H * dv)):
            mat(f"{t}.weight", n, d)
            vec(f"{t}.conv", (n, L), "n", 0.5)
        mat("b.weight", H, d)
        vec("A_log", (H,), "u", -2.0, 0.5), vec("norm.weight", (dv,), "u", 0.5, 1.5)
        mat("o.weight", d, H * dv)
        if part == "delta":
            mat("a.weight", H, d), mat("g.weight", H * dv, d)
            vec("dt_bias", (H,), "u", -1.0, 1.0)
        else:
            mat("a1.weight", R, d), mat("a2.weight", H * dk, R, 0.3), mat("g1.weight", R, d), mat("g2.weight", H * dv, R, 0.3)
            vec("dt_bias", (H * dk,), "u", -1.0, 1.0)
        return "mixer", PartSpec.make("gated_delta", size=d, heads=H, kv_heads=G, key_dim=dk, value_dim=dv, taps=L, norm_eps=EPS,
                                      decay="head" if part == "delta" else "channel",
                                      gate="silu" if part == "delta" else "sigmoid_lowrank"), W
    if part == "parallel":
        H, G, hd, R = d // 64, d // 128, 64, 16
        left = PartSpec.make("attention", prefix="left.", size=d, heads=H, kv_heads=G, head_dim=hd, v_dim=hd, qk_norm=False,
                             norm_eps=EPS, position=PartSpec.make("none"), window=None, scale=0.125, softcap=30.0, chunk=1024, head_gate=True)
        right = PartSpec.make("time_mix", prefix="right.", size=d, heads=H, key_dim=hd, norm_eps=EPS)
        p = "left."
        mat(p + "q_proj.weight", H * hd, d), mat(p + "k_proj.weight", G * hd, d), mat(p + "v_proj.weight", G * hd, d)
        mat(p + "gate.weight", H, d), mat(p + "out_proj.weight", d, H * hd)
        p = "right."
        for s in "rkvgw":
            vec(p + "mu." + s, (d,), "u", 0.0, 1.0)
        for s in "rkvg":
            mat(p + s + ".weight", H * hd, d)
        mat(p + "w1.weight", R, d), mat(p + "w2.weight", H * hd, R, 0.3)
        vec(p + "w0", (H * hd,), "u", -3.0, 0.0), vec(p + "u", (H, hd), "n", 0.5), vec(p + "norm.weight", (H * hd,), "u", 0.5, 1.5)
        mat(p + "o.weight", d, H * hd)
        vec("out.0.weight", (d,), "u", 0.5, 1.5), vec("out.1.weight", (d,), "u", 0.5, 1.5)
        return "mixer", PartSpec.make("parallel", size=d, branches=(left, right), norm_eps=EPS), W
    if part == "hgrn2":
        H, dk, dv = d // 128, 128, 128
        mat("q.weight", H * dk, d), mat("f.weight", H * dk, d), mat("v.weight", H * dv, d), mat("o.weight", d, H * dv)
        vec("f.bias", (H * dk,), "n", 1.0), vec("lower", (H * dk,), "u", 0.0, 0.9), vec("norm.weight", (dv,), "u", 0.5, 1.5)
        return "mixer", PartSpec.make("hgrn2", size=d, heads=H, key_dim=dk, value_dim=dv, norm_eps=EPS), W
    if part == "latent":
        H, dn, dr, dv, rq, rk = d // 128, 128, 64, 128, d * 3 // 4, 512
        mat("dq.weight", rq, d), mat("uq.weight", H * (dn + dr), rq), mat("dkv.weight", rk + dr, d)
        mat("uk.weight", H * dn, rk), mat("uv.weight", H * dv, rk), mat("o.weight", d, H * dv)
        vec("dq.norm", (rq,), "u", 0.5, 1.5), vec("dkv.norm", (rk,), "u", 0.5, 1.5), vec("sink", (H,), "n", 1.0)
        s = SCALED
        return "mixer", PartSpec.make("latent_attention", size=d, heads=H, dim=dn, rot_dim=dr, v_dim=dv, q_rank=rq, kv_rank=rk,
                                      scale=192 ** -0.5, norm_eps=EPS, window=1024, sink=True,
                                      position=PartSpec.make("rope", rot_dim=dr, theta=10000.0, pairing="adjacent", table64=True,
                                                             scaling=(s["factor"], s["original"], s["fast"], s["slow"]))), W
    raise ValueError(part)


def weights(case, seed, layer):
    """{local name: tensor} in the engine's dtypes: matrices in the case's dtype, vectors float32."""
    g = _gen(seed, 1 + 16 * layer)
    out = {}
    for name, shape, kind, a, b in make(case)[2]:
        if kind == "m":
            out[name] = _normal(g, shape, a, getattr(torch, case["dtype"]))
        elif kind == "n":
            out[name] = _normal(g, shape, a, torch.float32)
        else:
            out[name] = _uniform(g, shape, a, b)
    return out


def inputs(case, seed, layer):
    """The step's normed rows [rows, width], and what the cache holds already: keys and values per request."""
    dt = getattr(torch, case["dtype"])
    h = _normal(_gen(seed, 2 + 16 * layer), (case["rows"], case["width"]), 1.0, dt)
    if not case["history"]:
        return h, None
    d, part = case["width"], case["part"]
    n = sum(histories(case))
    g = _gen(seed, 3 + 16 * layer)
    if part == "latent":
        return h, _normal(g, (n, 512 + 64), 1.0, dt)
    G = {"attention_lfm2": 8, "attention_samusun": d // 256, "attention_nalizen": d // 256}[part]
    return h, _normal(g, (n, G * 64 * (1 if part == "attention_samusun" else 2)), 1.0, dt)


def cache_layout(case):
    """(key heads, key size, value size kept beside the key) of an attention part's pages."""
    d, part = case["width"], case["part"]
    return {"latent": (1, 576, 0), "attention_lfm2": (8, 64, 64), "attention_samusun": (d // 256, 64, 0),
            "attention_nalizen": (d // 256, 64, 64)}[part]


# ----------------------------------------------------------------------------------------------------------- one part

class _Step:
    """A step's index arrays, as the engine's step function hands them to a part."""

    def __init__(self, slots, starts, lengths):
        i32 = dict(dtype=torch.int32, device=DEV)
        n, T = len(slots), sum(lengths)
        rows = [(i, s + t) for i, (s, l) in enumerate(zip(starts, lengths)) for t in range(l)]
        self.positions = torch.tensor([p for _, p in rows], **i32)
        self.row_item = torch.tensor([i for i, _ in rows], **i32)
        self.row_slot = torch.tensor([slots[i] for i, _ in rows], **i32)
        self.item_start = torch.tensor([sum(lengths[:i]) for i in range(n + 1)], **i32)
        self.item_slot = torch.tensor(slots, **i32)
        self.item_len = torch.tensor([s + l for s, l in zip(starts, lengths)], **i32)
        self.n_rows, self.n_items = T, n
        self.all_single, self.max_item_rows = T == n, max(lengths)
        self.max_len = max(s + l for s, l in zip(starts, lengths))
        self.status = torch.zeros(1, **i32)
        self.carried, self.host, self.fixed_addresses = {}, None, True


def _bind(part, w):
    kids = part.children()
    if not kids:
        part.bind(w)
        return
    for kid, prefix in zip(kids, ("left.", "right.")):
        kid.bind({n[len(prefix):]: t for n, t in w.items() if n.startswith(prefix)})
    part.bind({n: t for n, t in w.items() if not n.startswith(("left.", "right."))})


def _prepare_part(case, seed):
    dt = getattr(torch, case["dtype"])
    category, spec, _ = make(case)
    layers = range(case["layers"])
    parts = [build_part(category, spec, case["dtype"]) for _ in layers]
    for i, part in enumerate(parts):
        _bind(part, weights(case, seed, i))
    lengths, before = shares(case), histories(case)
    n_ctx = 8192
    room = sum(-(-(a + b) // PAGE) * PAGE for a, b in zip(lengths, before))
    needs = [part.cache_need() if category == "mixer" else None for part in parts]
    cache = CacheManager(needs, page_tokens=PAGE, max_tokens=room, max_requests=len(lengths), n_ctx=n_ctx, dtype=dt, device=DEV)
    for part in parts:
        for p in [part] + list(part.children()):
            p.reserve(torch.device(DEV, torch.cuda.current_device()), len(lengths), n_ctx)
    ops.register_weight_chain([w for part in parts for w in part.weight_order()])
    slots = []
    for i, (a, b) in enumerate(zip(lengths, before)):
        slots.append(cache.add_request(i))
        if b:
            cache.reserve(i, b)
            cache.advance(i, b)
        cache.reserve(i, a)
    cache.flush()
    ctx = _Step(slots, before, lengths)
    views = cache.views(ctx.item_slot)
    rows = []
    for i, view in enumerate(views):
        h, past = inputs(case, seed, i)
        rows.append(h)
        if past is not None:
            G, hd, vd = cache_layout(case)
            past_step = _Step(slots, [0] * len(slots), before)
            ops.kv_write(past, 0, G * hd if vd else 0, view.pool, view.block_table, past_step.positions, past_step.row_slot, view.layer,
                         PAGE, G, hd, vd, status=past_step.status)
    out = torch.empty((case["rows"], case["width"]), dtype=torch.float32, device=DEV)

    def one_pass():
        out.zero_()                       # parts add their results to the residual stream
        ctx.carried = {}
        for part, view, h in zip(parts, views, rows):
            if category == "mixer":
                part.forward(h, ctx, view, out)
            else:
                part.forward(h, ctx, out)

    one_pass()
    one_pass()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    collecting = gc.isenabled()
    gc.disable()                          # a collected graph would end the recording
    try:
        with torch.cuda.graph(graph):
            one_pass()
    finally:
        if collecting:
            gc.enable()
    for g in cache.fixed:
        g.states.zero_()
    torch.cuda.synchronize()
    kept = [g.pool for g in cache.paged] + [g.states for g in cache.fixed]
    return {"graph": graph, "outputs": {"out": out, **{f"kept{i}": t for i, t in enumerate(kept)}}, "alive": (parts, cache, ctx, rows)}


# -------------------------------------------------------------------------------------------------------- whole calls

def _lfm2_config(shape):
    width, heads, ff = SHAPES[shape]
    return dict(architectures=["Lfm2ForCausalLM"], vocab_size=VOCAB, hidden_size=width, num_hidden_layers=LAYERS,
                num_attention_heads=heads, num_key_value_heads=8, head_dim=64, full_attn_idxs=list(ATTENTION_LAYERS),
                block_ff_dim=ff, block_auto_adjust_ff_dim=False, rope_theta=1000000.0, rope_pairing="split_half", conv_L_cache=3,
                conv_bias=False, norm_eps=EPS, tie_word_embeddings=True, max_position_embeddings=128000)


def _lfm2_weights(shape, seed):
    """Normal matrices; what a layer adds to the stream starts small, as models are initialised: over sqrt(2 layers)."""
    d, H, ff = SHAPES[shape]
    small = 0.02 / math.sqrt(2 * LAYERS)
    g, bf = _gen(seed, 1), torch.bfloat16
    w = {"model.embed_tokens.weight": _normal(g, (VOCAB, d), 0.15, bf), "model.embedding_norm.weight": _uniform(g, (d,), 0.5, 1.5).to(bf)}
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        w[p + "operator_norm.weight"], w[p + "ffn_norm.weight"] = _uniform(g, (d,), 0.5, 1.5).to(bf), _uniform(g, (d,), 0.5, 1.5).to(bf)
        if i in ATTENTION_LAYERS:
            for name, n in (("q_proj", H * 64), ("k_proj", 8 * 64), ("v_proj", 8 * 64)):
                w[p + f"self_attn.{name}.weight"] = _normal(g, (n, d), 0.02, bf)
            w[p + "self_attn.out_proj.weight"] = _normal(g, (d, H * 64), small, bf)
            w[p + "self_attn.q_layernorm.weight"] = _uniform(g, (64,), 0.5, 1.5).to(bf)
            w[p + "self_attn.k_layernorm.weight"] = _uniform(g, (64,), 0.5, 1.5).to(bf)
        else:
            w[p + "conv.in_proj.weight"], w[p + "conv.out_proj.weight"] = _normal(g, (3 * d, d), 0.02, bf), _normal(g, (d, d), small, bf)
            w[p + "conv.conv.weight"] = _normal(g, (d, 1, 3), 0.5, bf)
        for name, shp, std in (("w1", (ff, d), 0.02), ("w3", (ff, d), 0.02), ("w2", (d, ff), small)):
            w[p + f"feed_forward.{name}.weight"] = _normal(g, shp, std, bf)
    return w


def _prompts(case, seed):
    """The prompts of every request and the tokens it decodes behind them, as a program has them: lists of ids."""
    g = torch.Generator()
    g.manual_seed(seed * 1009 + 5)
    pick = lambda n: torch.randint(0, VOCAB, (n,), generator=g).tolist()  # noqa: E731
    return [pick(max(2, n)) for n in shares(dict(case, rows=max(case["rows"], 2 * case["requests"])))], [pick(case["tokens"]) for _ in range(case["requests"])]


def _prepare_serve(case, seed):
    from fellm_b200.config import EngineOptions
    from fellm_b200.config.registry import config_from_dict
    from fellm_b200.engine import Engine
    arch, config = config_from_dict(_lfm2_config(case["shape"]))
    prompts, follow = _prompts(case, seed)
    n = case["requests"]
    options = EngineOptions(dtype="bfloat16", n_ctx=4096, max_requests=max(n, 8), max_tokens=sum(len(p) for p in prompts) + n * (case["tokens"] + 2 * PAGE),
                            n_batch=4096)
    return {"engine": Engine(arch, config, options, tensors=_lfm2_weights(case["shape"], seed)), "prompts": prompts, "follow": follow}


def _run_serve(state):
    from fellm_b200.engine import StepItem
    engine, out = state["engine"], []
    for r in range(len(state["prompts"])):
        engine.add_request(r)
    out.append(engine.step([StepItem(r, p, [len(p) - 1]) for r, p in enumerate(state["prompts"])]))
    for t in range(len(state["follow"][0])):
        out.append(engine.step([StepItem(r, [f[t]], [0]) for r, f in enumerate(state["follow"])]))
    for r in range(len(state["prompts"])):
        engine.release(r)
    return out


# ------------------------------------------------------------------------------------------------ what a measurer calls

def prepare(case, seed):
    return _prepare_serve(case, seed) if case["part"] == "serve" else _prepare_part(case, seed)


def run(state):
    if "engine" in state:
        return _run_serve(state)
    state["graph"].replay()
    return state["outputs"]


def work(case):
    part = case["part"]
    if part == "serve":
        d, H, ff = SHAPES[case["shape"]]
        n, k = case["requests"], case["tokens"]
        R = max(case["rows"], 2 * n)
        conv, att = LAYERS - len(ATTENTION_LAYERS), len(ATTENTION_LAYERS)
        body = conv * 4 * d * d + att * (2 * d * H * 64 + 2 * d * 512) + LAYERS * 3 * d * ff
        kv = att * 2 * 512 * 2
        bytes_ = (1 + k) * 2 * (body + VOCAB * d) + kv * (R + k * R + n * k * k // 2) + (1 + k) * n * VOCAB * 4
        return {"bytes": bytes_, "flops": 2 * body * (R + n * k) + 2 * VOCAB * d * n * (1 + k) + att * 2 * 64 * H * sum(m * m for m in shares(dict(case, rows=R)))}
    e = 2 if case["dtype"] == "bfloat16" else 4
    d, R, n = case["width"], case["rows"], case["requests"]          # (of one layer; times the layers at the end)
    mats = [(name, shape) for name, shape, kind, _, _ in make(case)[2] if kind == "m"]
    size = sum(math.prod(s) for _, s in mats)
    flops, bytes_ = 2 * R * size, size * e + R * d * (e + 4)
    if part == "experts":                 # a token uses two of twelve choices, eight of which have matrices
        one = 3 * d * {1024: 3328, 2048: 6144}[d]
        pairs = 2 * R * 8 / 12
        bytes_ = e * one * 8 * (1 - (7 / 8) ** pairs) + R * d * (e + 4)
        flops = 2 * pairs * one
    if part in RECURRENT:
        H, dk = (d // 64, 64) if part == "parallel" else (d // 128, 128)
        flops += R * H * dk * dk * (8 if "delta" in part else 6)
        bytes_ += 2 * n * H * dk * dk * 4
    if part.startswith("attention") or part in ("latent", "parallel"):
        G, hd, vd = cache_layout(case) if part != "parallel" else (d // 128, 64, 64)
        H, window = (d // 128 if part == "latent" else d // 64), (4096 if part == "attention_lfm2" else 1024)
        seen = lambda a, b: sum(min(window, b + t + 1) for t in range(a))  # noqa: E731
        reads = [(a, b) for a, b in zip(shares(case), histories(case))]
        pairs = sum(seen(a, b) for a, b in reads)
        bytes_ += e * G * (hd + vd) * sum(min(b, window) + a for a, b in reads)
        flops += 2 * pairs * H * (320 if part == "latent" else 128)         # (a head's scores and sums, the latents expanded)
    return {"bytes": bytes_ * case["layers"], "flops": flops * case["layers"]}


def tolerance(case):
    """About four times what a comparison with exact() shows: rounded inputs to the products and rounded activations in
    16 bits; sums in another order in 32 bits; in whole calls, sixteen layers of it."""
    if case["part"] == "serve":
        return {"rel": 0.03, "max": 0.3}
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-3}
    return {"rel": 0.015, "max": 0.3}


# ------------------------------------------------------------------------------------------- the same in 64-bit numbers

def _unit(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(pos, freqs):
    """Angles are products of 32-bit numbers in this engine; cosines and sines of them in 64 bits."""
    a = (pos.to(torch.float32)[:, None] * torch.tensor(freqs, dtype=torch.float64).to(torch.float32).to(DEV)[None, :]).double()
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _rotate_halves(x, pos, freqs):
    """x [T, heads, size]: element i with i + len(freqs), the rest as it is."""
    m = len(freqs)
    c, s = _angles(pos, freqs)
    u, v = x[..., :m], x[..., m:2 * m]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * m:]], -1)


def _rotate_pairs(x, pos, freqs, mag):
    c, s = _angles(pos, freqs)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([(u * c - v * s) * mag, (v * c + u * s) * mag], -1).flatten(-2)


def _base_freqs(dims, base):
    return [base ** (-2.0 * i / dims) for i in range(dims // 2)]


def _scaled_freqs(dims, base):
    f, s = _base_freqs(dims, base), SCALED
    at = lambda turns: dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(at(s["fast"])), 0), min(math.ceil(at(s["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(len(f))]
    return [x / s["factor"] * r + x * (1 - r) for x, r in zip(f, ramp)], 0.1 * math.log(s["factor"]) + 1.0


def _band_freqs(dims, base):
    out, b = [], BANDS
    for f in _base_freqs(dims, base):
        wl = 2 * math.pi / f
        if wl < b["original"] / b["high"]:
            out.append(f)
        elif wl > b["original"] / b["low"]:
            out.append(f / b["factor"])
        else:
            s = (b["original"] / wl - b["low"]) / ((b["high"] - b["low"]) or 1.0)
            out.append((1 - s) * f / b["factor"] + s * f)
    return out


def _attend(q, k, v, first, scale, see, bias=None, cap=None, sink=None):
    """q [T, H, dk] at positions first..; k, v [first + T, G, .]; see(i, j): what a query at i reads."""
    T, H, _ = q.shape
    G = k.shape[1]
    i = (torch.arange(T, device=DEV) + first)[:, None]
    j = torch.arange(first + T, device=DEV)[None, :]
    mask = (j <= i) & see(i, j)
    out = torch.empty((T, H, v.shape[2]), dtype=torch.float64, device=DEV)
    for h in range(H):
        s = q[:, h] @ k[:, h // (H // G)].T * scale
        if bias is not None:
            s = s - bias[h] * (i - j)
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~mask, -math.inf)
        m = s.max(-1, keepdim=True).values
        if sink is not None:
            m = m.clamp(min=float(sink[h]))
        p = torch.exp(s - m)
        total = p.sum(-1, keepdim=True) + (torch.exp(sink[h] - m) if sink is not None else 0.0)
        out[:, h] = (p / total) @ v[:, h // (H // G)]
    return out


def _conv_silu(x, taps):
    L = taps.shape[1]
    xp = torch.cat([x.new_zeros(L - 1, x.shape[1]), x], 0)
    return F.silu(sum(xp[j:j + x.shape[0]] * taps[:, j] for j in range(L)))


def _delta(h, w, case):
    d, channel = case["width"], case["part"] == "channel_delta"
    H, G, dk, dv, T = d // 128, d // 256, 128, 128, h.shape[0]
    q, k, v = (_conv_silu(h @ w[f"{t}.weight"].T, w[f"{t}.conv"]).view(T, -1, 128) for t in "qkv")
    q = (q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5).repeat_interleave(H // G, 1)
    k = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    beta, rate = torch.sigmoid(h @ w["b.weight"].T), torch.exp(w["A_log"])
    if channel:
        a = ((h @ w["a1.weight"].T) @ w["a2.weight"].T + w["dt_bias"]).view(T, H, dk)
        g = torch.exp(-rate[None, :, None] * F.softplus(a))
        gate = torch.sigmoid((h @ w["g1.weight"].T) @ w["g2.weight"].T)
    else:
        g = torch.exp(-rate * F.softplus(h @ w["a.weight"].T + w["dt_bias"]))[:, :, None].expand(T, H, dk)
        gate = F.silu(h @ w["g.weight"].T)
    S, o = h.new_zeros(H, dk, dv), h.new_empty(T, H, dv)
    for t in range(T):
        S = S * g[t][:, :, None]
        u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None]
        o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return (_unit(o, EPS) * w["norm.weight"]).reshape(T, -1) * gate @ w["o.weight"].T, S


def _hgrn2(h, w, case):
    T, H = h.shape[0], case["width"] // 128
    q = F.silu(h @ w["q.weight"].T).view(T, H, 128)
    f = (w["lower"] + (1 - w["lower"]) * torch.sigmoid(h @ w["f.weight"].T + w["f.bias"])).view(T, H, 128)
    v = (h @ w["v.weight"].T).view(T, H, 128)
    S, o = h.new_zeros(H, 128, 128), h.new_empty(T, H, 128)
    for t in range(T):
        S = f[t][:, :, None] * S + (1 - f[t])[:, :, None] * v[t][:, None]
        o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return (_unit(o, EPS) * w["norm.weight"]).reshape(T, -1) @ w["o.weight"].T, S


def _parallel(h, w, case):
    d, T = case["width"], h.shape[0]
    H, G = d // 64, d // 128
    p = "left."
    q, k, v = (h @ w[p + f"{t}_proj.weight"].T for t in "qkv")
    left = _attend(q.view(T, H, 64), k.view(T, G, 64), v.view(T, G, 64), 0, 0.125, lambda i, j: i // 1024 == j // 1024, cap=30.0)
    left = (left * torch.sigmoid(h @ w[p + "gate.weight"].T)[:, :, None]).reshape(T, -1) @ w[p + "out_proj.weight"].T
    p = "right."
    prev = torch.cat([h.new_zeros(1, d), h[:-1]], 0)
    r, k, v, g, z = (h + (prev - h) * w[p + "mu." + s] for s in "rkvgw")
    r, k, v = ((x @ w[p + s + ".weight"].T).view(T, H, 64) for x, s in ((r, "r"), (k, "k"), (v, "v")))
    gate = F.silu(g @ w[p + "g.weight"].T)
    decay = torch.exp(-torch.exp(torch.tanh(z @ w[p + "w1.weight"].T) @ w[p + "w2.weight"].T + w[p + "w0"])).view(T, H, 64)
    S, o = h.new_zeros(H, 64, 64), h.new_empty(T, H, 64)
    for t in range(T):
        kv = k[t][:, :, None] * v[t][:, None]
        o[t] = torch.bmm(r[t][:, None], S + w[p + "u"][:, :, None] * kv)[:, 0]
        S = decay[t][:, :, None] * S + kv
    right = (_unit(o, EPS).reshape(T, -1) * w[p + "norm.weight"] * gate) @ w[p + "o.weight"].T
    return 0.5 * (_unit(left, EPS) * w["out.0.weight"] + _unit(right, EPS) * w["out.1.weight"]), S


def _latent(h, w, case, past, first):
    H, T = case["width"] // 128, h.shape[0]
    pos = torch.arange(T, device=DEV) + first
    q = ((_unit(h @ w["dq.weight"].T, EPS) * w["dq.norm"]) @ w["uq.weight"].T).view(T, H, 192)
    kv = h @ w["dkv.weight"].T
    freqs, mag = _scaled_freqs(64, 10000.0)
    new = torch.cat([_unit(kv[:, :512], EPS) * w["dkv.norm"], _rotate_pairs(kv[:, None, 512:], pos, freqs, mag)[:, 0]], -1)
    rows = new if past is None else torch.cat([past, new], 0)
    n = rows.shape[0]
    k = torch.cat([(rows[:, :512] @ w["uk.weight"].T).view(n, H, 128), rows[:, None, 512:].expand(n, H, 64)], -1)
    v = (rows[:, :512] @ w["uv.weight"].T).view(n, H, 128)
    q = torch.cat([q[..., :128], _rotate_pairs(q[..., 128:], pos, freqs, mag)], -1)
    o = _attend(q, k, v, first, 192 ** -0.5, lambda i, j: i - j < 1024, sink=w["sink"])
    return o.reshape(T, -1) @ w["o.weight"].T


def _attention(h, w, case, past, first):
    d, T, part = case["width"], h.shape[0], case["part"]
    H = d // 64
    G, _, vd = cache_layout(case)
    pos = torch.arange(T, device=DEV) + first
    q, k = h @ w["q_proj.weight"].T, h @ w["k_proj.weight"].T
    see, bias, gate = (lambda i, j: i - j < 1024), None, None
    if part == "attention_samusun":
        temp = 1 + 0.25 * torch.log(torch.floor((pos.double() + 1) / 128) + 1)
        q, k = (q + w["q_proj.bias"]).view(T, H, 64) * temp[:, None, None], (k + w["k_proj.bias"]).view(T, G, 64)
        v, bias = k, [2.0 ** (-8.0 * (i + 1) / H) for i in range(H)]
    else:
        q, k, v = q.view(T, H, 64), k.view(T, G, 64), (h @ w["v_proj.weight"].T).view(T, G, 64)
        if part == "attention_lfm2":
            freqs = (torch.tensor(1000000.0) ** (-(2.0 * torch.arange(32, dtype=torch.float32)) / 64.0)).double().tolist()
            q, k = (_rotate_halves(_unit(x, EPS) * w[n + "_norm.weight"], pos, freqs) for x, n in ((q, "q"), (k, "k")))
            see = lambda i, j: j <= i  # noqa: E731
        else:
            freqs = _band_freqs(32, 10000.0)
            q, k = (_unit(_rotate_halves(x, pos, freqs), EPS) for x in (q, k))
            gate = torch.sigmoid(h @ w["out_gate.weight"].T)
    if past is not None:
        n = G * 64
        k = torch.cat([past[:, :n].view(-1, G, 64), k], 0)
        v = torch.cat([past[:, n:].view(-1, G, 64), v], 0) if vd else k
    o = _attend(q, k, v, first, 0.125, see, bias=bias).reshape(T, -1)
    if gate is not None:
        o = o * gate
    return o @ w["out_proj.weight"].T + (w["out_proj.bias"] if bias is not None else 0.0)


def _experts(h, w, case):
    s = torch.softmax(h @ w["router.weight"].T, -1)
    c = s + w["correction"]
    T, n = c.shape
    best = c.view(T, 4, n // 4).max(-1).values.topk(2, -1).indices
    keep = torch.zeros((T, 4), dtype=torch.bool, device=DEV).scatter_(1, best, True).repeat_interleave(n // 4, 1)
    chosen = c.masked_fill(~keep, -math.inf).topk(2, -1).indices
    out = torch.zeros_like(h)
    for e in range(n):
        rows = (chosen == e).any(-1).nonzero()[:, 0]
        x = h[rows]
        y = x if e >= 8 else (F.silu(x @ w[f"e{e}.gate.weight"].T) * (x @ w[f"e{e}.up.weight"].T)) @ w[f"e{e}.down.weight"].T
        out[rows] += s[rows, e][:, None] * y
    return out


def _exact_serve(case, seed):
    w = {n: t.double() for n, t in _lfm2_weights(case["shape"], seed).items()}
    prompts, follow = _prompts(case, seed)
    d, H, _ = SHAPES[case["shape"]]
    freqs = (torch.tensor(1000000.0) ** (-(2.0 * torch.arange(32, dtype=torch.float32)) / 64.0)).double().tolist()
    per_request = []
    for p, f in zip(prompts, follow):
        ids = torch.tensor(p + f, device=DEV)
        T, x = len(ids), w["model.embed_tokens.weight"][ids]
        pos = torch.arange(T, device=DEV)
        for i in range(LAYERS):
            n = f"model.layers.{i}."
            h = _unit(x, EPS) * w[n + "operator_norm.weight"]
            if i in ATTENTION_LAYERS:
                q, k, v = ((h @ w[n + f"self_attn.{t}_proj.weight"].T).view(T, -1, 64) for t in "qkv")
                q = _rotate_halves(_unit(q, EPS) * w[n + "self_attn.q_layernorm.weight"], pos, freqs)
                k = _rotate_halves(_unit(k, EPS) * w[n + "self_attn.k_layernorm.weight"], pos, freqs)
                x = x + _attend(q, k, v, 0, 0.125, lambda i, j: j <= i).reshape(T, -1) @ w[n + "self_attn.out_proj.weight"].T
            else:
                B, C, X = (h @ w[n + "conv.in_proj.weight"].T).split(d, 1)
                taps = w[n + "conv.conv.weight"].view(d, 3)
                bx = torch.cat([h.new_zeros(2, d), B * X], 0)
                x = x + (C * sum(bx[j:j + T] * taps[:, j] for j in range(3))) @ w[n + "conv.out_proj.weight"].T
            h = _unit(x, EPS) * w[n + "ffn_norm.weight"]
            x = x + (F.silu(h @ w[n + "feed_forward.w1.weight"].T) * (h @ w[n + "feed_forward.w3.weight"].T)) @ w[n + "feed_forward.w2.weight"].T
        per_request.append((_unit(x[len(p) - 1:], EPS) * w["model.embedding_norm.weight"]) @ w["model.embed_tokens.weight"].T)
    return [torch.stack([r[t] for r in per_request]) for t in range(case["tokens"] + 1)]


def _exact_layer(case, seed, layer):
    """(a layer's result, its requests' matrices after the step or None)."""
    part = case["part"]
    w = {n: t.double() for n, t in weights(case, seed, layer).items()}
    h, past = inputs(case, seed, layer)
    h, past = h.double(), None if past is None else past.double()
    if part == "swiglu":
        return (F.silu(h @ w["gate.weight"].T) * (h @ w["up.weight"].T)) @ w["down.weight"].T, None
    if part == "experts":
        return _experts(h, w, case), None
    outs, states, at, old = [], [], 0, 0
    for n, first in zip(shares(case), histories(case)):
        x, p = h[at:at + n], None if past is None else past[old:old + first]
        at, old = at + n, old + first
        if part in RECURRENT:
            y, S = (_delta if "delta" in part else _hgrn2 if part == "hgrn2" else _parallel)(x, w, case)
            states.append(S)
        else:
            y = (_latent if part == "latent" else _attention)(x, w, case, p, first)
        outs.append(y)
    return torch.cat(outs, 0), torch.stack(states) if states else None


def exact(case, seed):
    if case["part"] == "serve":
        return _exact_serve(case, seed)
    outs, states = zip(*(_exact_layer(case, seed, i) for i in range(case["layers"])))
    got = {"out": sum(outs)}
    if states[0] is not None:
        # states [slots and one row that belongs to nobody, layers, heads, .., ..]; the engine keeps a head's matrix column by column
        S = torch.stack(states, 1)
        S = S.transpose(-1, -2).reshape(S.shape)
        got[{"delta": "kept1", "channel_delta": "kept1", "parallel": "kept2", "hgrn2": "kept0"}[case["part"]]] = torch.cat([S, torch.zeros_like(S[:1])], 0)
    return got
