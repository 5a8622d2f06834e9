"""Cases by which the speed of the framework's main paths is followed: model steps and prompts, the acceptance rule, and
the fp32 backend operators, through their public entry points.

A case names its kind and sizes.  `prepare` makes what a program holds before the call (weights loaded once per model,
caches with their contexts, tokens on the device), `run` is one pass, `exact` the same outputs in 64 bits from plain torch.
"""

import math

import numpy as np
import torch

import versenext_b200 as vn
from versenext_b200 import sampling
from versenext_b200 import synthetic as S
from versenext_b200.device import DeviceArray

F = torch.float64
# 16 nodes: four children of the last committed token, two below each, two below the first two of those
TREE = [-1] * 4 + [0, 0, 1, 1, 2, 2, 3, 3] + [4, 4, 5, 5]


# ---- the cases ------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one verification step of the CPU-sized model (dim 64, two layers) in the default float32: launches and latency
        {"name": "small_f32_step", "kind": "verse", "model": "small", "dtype": "f32", "batch": 1, "new": 5, "ctx": 32},
        # one token of one request on the mate-shaped target: interactive decoding
        {"name": "mate_decode_1", "kind": "verse", "model": "mate", "dtype": "bf16", "batch": 1, "new": 1, "ctx": 511},
        # the verification step of the speculative workload: 32 requests, k = 4
        {"name": "mate_verify_32x5", "kind": "verse", "model": "mate", "dtype": "bf16", "batch": 32, "new": 5, "ctx": 512},
        # tree verification: 8 requests, 16 nodes, a context of 2048
        {"name": "mate_tree_8x16", "kind": "verse", "model": "mate", "dtype": "bf16", "batch": 8, "new": 16, "ctx": 2048, "tree": True},
        # the prompts of that workload's first step
        {"name": "mate_prompt_8x512", "kind": "verse", "model": "mate", "dtype": "bf16", "batch": 8, "new": 512, "ctx": 0},
        # quantised serving: INT4 with groups of 128, k = 6
        {"name": "mate_int4_verify_64x7", "kind": "verse", "model": "mate", "dtype": "bf16", "quant": "int4g128", "batch": 64, "new": 7, "ctx": 256},
        # a prompt of the two-layer draft-sized model in the default float32
        {"name": "draft_f32_prompt_2x300", "kind": "verse", "model": "draft", "dtype": "f32", "batch": 2, "new": 300, "ctx": 0},
        # a composed model: ragged prompts through latent attention, selective scan and delta rule layers
        {"name": "fuzudra_prompt_4x777", "kind": "fuzudra", "width": 1024, "batch": 4, "new": 777, "ctx": 0},
        # a composed model over several residual streams: one token of 32 requests
        {"name": "musutar_decode_32", "kind": "musutar", "width": 2048, "batch": 32, "new": 1, "ctx": 1000},
        # acceptance of 64 drafts of 4 tokens over the full vocabulary
        {"name": "accept_64x4", "kind": "accept", "batch": 64, "k": 4, "vocab": 248320, "temperature": 1.0, "top_k": 0},
        # the backend plugin's linear and attention on a transformer layer's activations
        {"name": "backend_linear", "kind": "linear", "rows": 1000, "in": 1024, "out": 2752},
        {"name": "backend_attention", "kind": "attention", "heads": 32, "queries": 500, "keys": 500, "dim": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "prompt", "prompt", "composed", "composed", "accept", "linear", "attention"])
    if kind == "step":
        if rng.random() < 0.25:
            return {"kind": "verse", "model": rng.choice(["small", "draft"]), "dtype": "f32", "batch": _log(rng, 1, 16), "new": rng.randint(1, 7),
                    "ctx": _log(rng, 8, 200)}
        if rng.random() < 0.2:
            return {"kind": "verse", "model": "mate", "dtype": "bf16", "batch": rng.randint(1, 8), "new": 16, "ctx": _log(rng, 64, 2048), "tree": True}
        c = {"kind": "verse", "model": "mate", "dtype": "bf16", "batch": _log(rng, 1, 64), "new": rng.randint(1, 7), "ctx": _log(rng, 32, 1024)}
        if rng.random() < 0.4:
            c["quant"] = rng.choice(["int8", "int4g128"])
        return c
    if kind == "prompt":
        if rng.random() < 0.3:
            return {"kind": "verse", "model": "draft", "dtype": "f32", "batch": rng.randint(1, 4), "new": _log(rng, 20, 300), "ctx": 0}
        return {"kind": "verse", "model": "mate", "dtype": "bf16", "batch": rng.randint(1, 4), "new": _log(rng, 33, 1024), "ctx": 0}
    if kind == "composed":
        c = {"kind": rng.choice(["fuzudra", "musutar"]), "width": rng.choice([1024, 2048])}
        if rng.random() < 0.5:
            return dict(c, batch=rng.randint(1, 2), new=_log(rng, 33, 777), ctx=0)
        return dict(c, batch=_log(rng, 1, 32), new=rng.randint(1, 3), ctx=_log(rng, 40, 400))
    if kind == "accept":
        return {"kind": "accept", "batch": _log(rng, 1, 64), "k": rng.randint(1, 6 if rng.random() < 0.3 else 4), "vocab": rng.choice([32000, 50257, 100003, 151936]),
                "temperature": rng.choice([0.8, 1.0]), "top_k": rng.choice([0, 50])}
    if kind == "linear":
        return {"kind": "linear", "rows": _log(rng, 1, 1000), "in": rng.choice([256, 509, 1000, 1024]), "out": rng.choice([256, 1023, 1024, 2752])}
    n = _log(rng, 16, 500)
    return {"kind": "attention", "heads": rng.randint(1, 32), "queries": rng.choice([1, n]), "keys": n, "dim": rng.choice([32, 64, 128])}


# ---- weights and models ---------------------------------------------------------------------------------------------
VERSE = {
    "small": dict(vocab_size=256, dim=64, n_layer=2, n_head=4, max_seq_len=512),
    "draft": dict(vocab_size=32000, dim=256, n_layer=2, n_head=4, max_seq_len=2048),
    "mate": dict(vocab_size=32000, dim=1024, n_layer=4, n_head=16, n_kv_head=8, layer_pattern=["mod", "trisparse", "trisparse", "trisparse"],
                 window_size=1024, num_global_tokens=128, use_alibi=False, use_rope=True, max_seq_len=4096, num_dense_parts=4, num_experts_per_part=4,
                 top_k=2, tie_weights=True, embedding_scale=True),
}
_COMPOSED = {"fuzudra": (vn.FuzudraLM, S.fuzudra_config, S.fuzudra_shapes), "musutar": (vn.MusutarLM, S.musutar_config, S.musutar_shapes)}
# (name's end, standard deviation, mean) of the composed models' tensors that are not plain linear weights
_SPECIAL = (("mix.A_log", 1.0, -1.0), ("mix.dt_bias", 1.0, -2.0), ("mix.dt.b", 1.0, -3.0), ("mix.D", 0.1, 1.0), ("mix.sink", 1.0, 0.0), (".conv", 0.4, 0.0),
            ("canon1", 0.3, 0.0), ("mix.norm", 0.1, 1.0), ("dkv.norm", 0.1, 1.0), ("hc1.in", 0.1, 0.25), ("hc2.in", 0.1, 0.25), ("hc1.out", 0.1, 1.0),
            ("hc2.out", 0.1, 1.0))


def _randn(shape, g, std, mean=0.0):
    return (torch.randn(shape, generator=g, device="cuda") * std + mean).bfloat16().float()


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _verse_weights(kw):
    """(name, float32 tensor holding bf16 values) in a fixed order."""
    g, rs = _gen(17), (2 * kw["n_layer"]) ** -0.5
    for name, shape in S._shapes(kw):
        if name.endswith(("norm1.weight", "norm2.weight")) or name == "norm.weight":
            yield name, _randn(shape, g, 0.1, 1.0)
        elif name.endswith("gate_logits"):
            yield name, _randn(shape, g, 0.5)
        else:
            yield name, _randn(shape, g, 0.02 * (rs if name.endswith(("attn.proj.weight", "ffn.w_down.weight")) else 1.0))


def _composed_weights(kind, cfg):
    g = _gen(19)
    for name, shape in _COMPOSED[kind][2](cfg).items():
        std, mean = (0.02, 0.0) if len(shape) == 2 else (0.1, 0.0)
        for end, s, m in _SPECIAL:
            if name.endswith(end):
                std, mean = s, m
        if kind == "musutar" and name.split(".")[-1] in ("norm", "norm1", "norm2"):
            mean = 1.0
        w = _randn(shape, g, std, mean)
        yield name, w + torch.eye(shape[0], device="cuda") if name.endswith(".mix") else w


_models = {}


def _model(case):
    """A loaded model: a program loads one when it starts and keeps it.  The last three used are kept here."""
    key = (case["kind"], case.get("model"), case.get("dtype"), case.get("quant"), case.get("width"))
    m = _models.pop(key, None)
    if m is None:
        if case["kind"] == "verse":
            kw = VERSE[case["model"]]
            m = vn.VerseNexLM(dtype=case["dtype"], **kw)
            for name, w in _verse_weights(kw):
                m.load_tensor(name, w.cpu().numpy())
            m.finalize()
            if case.get("quant"):
                m.quantize(case["quant"])
        else:
            cls, config, shapes = _COMPOSED[case["kind"]]
            cfg = config(case["width"])
            m = cls(cfg, shapes(cfg), dtype="bf16")
            for name, w in _composed_weights(case["kind"], cfg):
                m.load_tensor(name, w.cpu().numpy())
            m.finalize()
        while len(_models) > 2:
            _models.pop(next(iter(_models)))
    _models[key] = m
    return m


def _vocab(case):
    return VERSE[case["model"]]["vocab_size"] if case["kind"] == "verse" else 32000


def _lens(case):
    """Tokens that each request of a prompt brings: composed models take them ragged."""
    n, b = case["new"], case["batch"]
    return [n] * b if case["kind"] == "verse" or case["ctx"] else [max(1, n - (n * i) // (2 * b)) for i in range(b)]


def _tokens(case, seed):
    g = np.random.default_rng(seed)
    return g.integers(0, _vocab(case), (case["batch"], case["ctx"] + case["new"]))


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _accept_inputs(case, seed):
    B, k, V = case["batch"], case["k"], case["vocab"]
    g = _gen(seed)
    q = torch.randn((B, k, V), generator=g, device="cuda") * 2.0
    p = torch.empty((B, k + 1, V), device="cuda")
    p[:, :k] = q + torch.randn((B, k, V), generator=g, device="cuda") * 0.5
    p[:, k] = torch.randn((B, V), generator=g, device="cuda") * 2.0
    # tokens drawn from the draft's distribution
    noise = -torch.log(-torch.log(torch.rand((B, k, V), generator=g, device="cuda").clamp_(1e-9, 1 - 1e-6)))
    draft = torch.argmax(_kept(q / case["temperature"], case["top_k"]) + noise, -1)
    ua, us = torch.rand((B, k), generator=g, device="cuda"), torch.rand((B, k + 1), generator=g, device="cuda")
    return p, q, draft, ua, us


def _kept(x, top_k):
    if not top_k:
        return x
    return torch.where(x >= torch.topk(x, top_k, dim=-1).values[..., -1:], x, float("-inf"))


def _floats(case, seed):
    g = _gen(seed)
    if case["kind"] == "linear":
        return (torch.randn((case["rows"], case["in"]), generator=g, device="cuda"), torch.randn((case["out"], case["in"]), generator=g, device="cuda") * 0.02,
                torch.randn(case["out"], generator=g, device="cuda") * 0.1)
    shape = lambda n: (case["heads"], n, case["dim"])  # noqa: E731
    return tuple(torch.randn(shape(n), generator=g, device="cuda") for n in (case["queries"], case["keys"], case["keys"]))


def _device(t):
    """A torch tensor as an array of the library: the same memory."""
    return DeviceArray(vn.Context.get(0), t.data_ptr(), tuple(t.shape), np.int64 if t.dtype == torch.int64 else np.float32, base=t)


def _torch(a):
    return torch.as_tensor(a, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "accept":
        p, q, draft, ua, us = _accept_inputs(case, seed)
        return {"case": case, "in": [_device(x) for x in (p, q, draft, ua, us)]}
    if kind in ("linear", "attention"):
        return {"case": case, "op": vn.get_backend("cuda"), "in": [_device(x) for x in _floats(case, seed)]}
    m, B, ctx = _model(case), case["batch"], case["ctx"]
    toks = _tokens(case, seed)
    cache = m.new_cache(B, ctx + case["new"] + 8, max_pending=max(1, case["new"] if ctx else 1))
    part = max(1, 8192 // B)
    for lo in range(0, ctx, part):
        n = min(part, ctx - lo)
        m.forward_cached(toks[:, lo:lo + n], cache, want_logits=False, want_hidden=True, last_only=True)
        cache.commit(n, np.full(B, n, np.int32))
    s = {"case": case, "model": m, "cache": cache}
    lens = _lens(case)
    if kind != "verse" and not ctx:
        s.update(slots=np.arange(B, dtype=np.int32), counts=np.asarray(lens, np.int32), rows=np.cumsum(lens) - 1,
                 tokens=m.ctx.from_numpy(np.concatenate([toks[b, :n] for b, n in enumerate(lens)])))
    else:
        s["tokens"] = m.ctx.from_numpy(toks[:, ctx:])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "accept":
        p, q, draft, ua, us = s["in"]
        n, t = sampling.accept(p.ctx, p, q, draft, u_accept=ua, u_sample=us, temperature=case["temperature"], top_k=case["top_k"])
        return {"len": _torch(n), "tokens": _torch(t)}
    if kind == "linear":
        return _torch(s["op"].linear(*s["in"]))
    if kind == "attention":
        return _torch(s["op"].attention(*s["in"]))
    m, cache = s["model"], s["cache"]
    if case["ctx"]:
        return _torch(m.forward_cached(s["tokens"], cache, parents=TREE if case.get("tree") else None))
    cache.reset()
    if kind == "verse":
        logits, hidden = m.forward_cached(s["tokens"], cache, last_only=True, want_hidden=True)
        return {"logits": _torch(logits), "hidden": _torch(hidden)}
    return _torch(m.forward_ragged(cache, s["slots"], s["counts"], s["tokens"], s["rows"]))


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _linear_sizes(case):
    """(weights read per pass, multiply-adds per token, head weights, width of keys and values, window, attention layers, heads x dim)"""
    if case["kind"] == "verse":
        kw = VERSE[case["model"]]
        D, H, G = kw["dim"], kw["n_head"], kw.get("n_kv_head") or kw["n_head"]
        head, total, per_token, tokens = kw["vocab_size"] * D, 0, 0, case["batch"] * case["new"]
        for name, shape in S._shapes(kw):
            n = int(np.prod(shape))
            if len(shape) != 2 or name == "tok_emb.weight" or "global_tokens" in name:
                continue
            share = kw["top_k"] / kw["num_experts_per_part"] if ".experts." in name else 1.0
            total += n * (1.0 - (1.0 - share) ** tokens)
            per_token += n * share
        return total, per_token, head, G * (D // H), kw.get("window_size", 512), kw["n_layer"], D
    cfg = _COMPOSED[case["kind"]][1](case["width"])
    D, head = case["width"], 32000 * case["width"]
    total = sum(int(np.prod(s)) for n, s in _COMPOSED[case["kind"]][2](cfg).items() if len(s) == 2 and n not in ("embed", "head"))
    return total, total, head, D // 4, 1024, 1 if case["kind"] == "fuzudra" else 2, D


def work(case):
    kind = case["kind"]
    if kind == "accept":
        n = case["batch"] * case["vocab"] * (2 * case["k"] + 1)
        return {"bytes": 4.0 * n, "flops": 4.0 * n}
    if kind == "linear":
        M, K, N = case["rows"], case["in"], case["out"]
        return {"bytes": 4.0 * (M * K + N * K + M * N), "flops": 2.0 * M * N * K}
    if kind == "attention":
        H, q, k, d = case["heads"], case["queries"], case["keys"], case["dim"]
        return {"bytes": 4.0 * H * d * 2 * (q + k), "flops": 4.0 * H * q * k * d}
    total, per_token, head, kv, window, layers, width = _linear_sizes(case)
    B, ctx = case["batch"], case["ctx"]
    tokens = sum(_lens(case))
    rows = B * case["new"] if ctx else B
    item = 4.0 if case.get("dtype") == "f32" else 2.0
    w_item = {"int8": 1.0, "int4g128": 0.5 + 2 / 128}.get(case.get("quant"), item)
    seen = min(ctx + case["new"], window)
    nbytes = (total + head) * w_item + layers * B * (min(ctx, window) + case["new"]) * 2 * kv * item + rows * _vocab(case) * 4.0
    pairs = tokens * (seen if ctx else seen / 2)
    return {"bytes": nbytes, "flops": 2.0 * tokens * per_token + 2.0 * rows * head + 4.0 * layers * pairs * width}


def tolerance(case):
    """About four times the distance from the 64-bit values: 16-bit operands and caches (0.0018 for the transformer models, 0.0055 for the composed ones),
    or 32-bit sums.  The acceptance rule's decisions have one answer."""
    if case["kind"] == "accept":
        return "exact"
    if case["kind"] in ("linear", "attention"):
        return {"rel": 3e-6, "max": 1e-4}
    if case.get("dtype") == "f32":
        return {"rel": 3e-6, "max": 1e-4}
    return {"rel": 8e-3, "max": 0.3} if case["kind"] == "verse" else {"rel": 2.2e-2, "max": 0.8}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _quantised(w, scheme):
    """Values that a weight-only quantised linear multiplies with."""
    w = w.float()
    if scheme == "int8":
        scale = (w.abs().amax(1, keepdim=True) / 127.0)
        return (torch.round(w / scale).clamp(-127, 127) * scale).to(F)
    n = w.shape[1]
    g = torch.nn.functional.pad(w, (0, -n % 128)).reshape(w.shape[0], -1, 128)
    scale = (g.abs().amax(2, keepdim=True) / 7.0).bfloat16().float()
    return (torch.round(g / scale).clamp(-8, 7) * scale).reshape(w.shape[0], -1)[:, :n].to(F)


def _exact_verse(case, seed):
    kw = VERSE[case["model"]]
    quant = case.get("quant")
    W = {}
    for name, w in _verse_weights(kw):
        dense = len(w.shape) != 2 or "router.gate" in name or "global_tokens" in name or name == "tok_emb.weight"
        W[name] = w.to(F) if dense or not quant else _quantised(w, quant)
    head = _quantised(W["tok_emb.weight"], quant) if quant else W["tok_emb.weight"]
    D, H = kw["dim"], kw["n_head"]
    G, hd = kw.get("n_kv_head") or H, D // H
    window, n_g = kw.get("window_size", 512), kw.get("num_global_tokens", 64)
    toks = torch.from_numpy(_tokens(case, seed)).cuda()
    B, ctx, new = case["batch"], case["ctx"], case["new"]
    T = ctx + new
    pos = torch.arange(T, device="cuda")
    seen = pos[None, :] <= pos[:, None]
    if case.get("tree"):
        depth, anc = [0] * new, torch.eye(new, dtype=torch.bool)
        for i, p in enumerate(TREE):
            if p >= 0:
                depth[i] = depth[p] + 1
                anc[i] |= anc[p]
        pos[ctx:] = ctx + torch.tensor(depth, device="cuda")
        seen[ctx:, ctx:] = anc.cuda()
    dist = pos[:, None] - pos[None, :]
    minus = -float("inf")
    in_window = torch.where(seen & (dist < window), 0.0, minus).to(F)
    slopes = 2.0 ** (-(torch.arange(1, H + 1, device="cuda", dtype=F) / H))

    def turn(x):                                            # [T, heads, hd]
        half = hd // 2
        freq = np.float32(1.0) / (np.float32(10000.0) ** (np.float32(2.0) * np.arange(half, dtype=np.float32) / np.float32(hd)))
        a = pos.to(F)[:, None] * torch.from_numpy(freq.astype(np.float64)).cuda()[None, :]
        c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
        u, v = x[..., :half], x[..., half:]
        return torch.cat([u * c - v * s, u * s + v * c], -1)

    def heads(x, n):
        return x.reshape(-1, n, hd)

    def attend(q, k, v, bias):
        k, v = (t.repeat_interleave(H // G, 1) for t in (k, v))
        s = torch.einsum("thd,shd->hts", q, k) * hd ** -0.5
        return torch.einsum("hts,shd->thd", torch.softmax(s if bias is None else s + bias, -1), v)

    def swiglu(x, p):
        return (torch.nn.functional.silu(x @ W[p + "w_gate.weight"].T) * (x @ W[p + "w_up.weight"].T)) @ W[p + "w_down.weight"].T

    x = W["tok_emb.weight"][toks] * (math.sqrt(D) if kw.get("embedding_scale") else 1.0)
    for i, kind in enumerate(kw.get("layer_pattern") or ["trisparse"] * kw["n_layer"]):
        p = f"blocks.{i}."
        h = _rms(x, W[p + "norm1.weight"], 1e-6)
        gate = torch.sigmoid(W[p + "attn.gate_logits"])
        wq, wk, wv = (W[p + f"attn.{n}.weight"] for n in ("wq", "wk", "wv"))
        sinks = W[p + "attn.global_tokens.weight"]
        sk, sv = heads(sinks @ wk.T, G), heads(sinks @ wv.T, G)
        out = []
        for b in range(B):
            q, k, v = heads(h[b] @ wq.T, H), heads(h[b] @ wk.T, G), heads(h[b] @ wv.T, G)
            if kw.get("use_rope"):
                q, k = turn(q), turn(k)
            o = gate[0] * attend(q, k, v, in_window) + gate[1] * attend(q, sk, sv, None)
            if kw.get("use_alibi", True):
                bias = torch.where(seen[None], -slopes[:, None, None] * dist.to(F), minus)
                o = o + gate[2] * attend(q, k, v, bias)
            out.append(o.reshape(T, D))
        x = x + torch.stack(out) @ W[p + "attn.proj.weight"].T
        h = _rms(x, W[p + "norm2.weight"], 1e-6)
        if kind != "mod":
            x = x + swiglu(h, p + "ffn.")
            continue
        f = h.reshape(-1, D)
        part = torch.softmax(f @ W[p + "ffn.part_router.gate.weight"].T, -1)
        y = torch.zeros_like(f)
        for a in range(kw["num_dense_parts"]):
            z = f @ W[p + f"ffn.parts.{a}.router.gate.weight"].T
            top = torch.topk(z, kw["top_k"], dim=-1)
            w = torch.zeros_like(z).scatter_(1, top.indices, torch.softmax(top.values, -1)) * part[:, a:a + 1]
            for e in range(kw["num_experts_per_part"]):
                at = torch.nonzero(w[:, e] > 0)[:, 0]
                y[at] += w[at, e:e + 1] * swiglu(f[at], p + f"ffn.parts.{a}.experts.{e}.")
        x = x + y.reshape(x.shape)
    hidden = _rms(x, W["norm.weight"], 1e-6)
    if ctx:
        return hidden[:, ctx:] @ head.T
    return {"logits": hidden[:, -1:] @ head.T, "hidden": hidden[:, -1:]}


def _conv(x, w, b=None):
    """Causal, per channel: x [B, T, C], w [C, taps]."""
    taps = w.shape[1]
    xp = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    y = sum(xp[:, j:j + x.shape[1]] * w[:, j] for j in range(taps))
    return y if b is None else y + b


def _window_attend(q, k, v, scale, window, sink=None):
    """q [B, T, H, d], k and v [B, T, G, .]: causal within a window; `sink` [H] joins the soft-max's sum."""
    T, H = q.shape[1:3]
    i = torch.arange(T, device="cuda")
    seen = (i[None, :] <= i[:, None]) & (i[:, None] - i[None, :] < (window or T))
    out = []
    for b in range(q.shape[0]):
        kb, vb = (t[b].repeat_interleave(H // t.shape[2], 1) for t in (k, v))
        s = torch.einsum("thd,shd->hts", q[b], kb) * scale
        s = torch.where(seen[None], s, -float("inf"))
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(-1, T, 1)], -1)
        out.append(torch.einsum("hts,shd->thd", torch.softmax(s, -1)[..., :T], vb))
    return torch.stack(out)


def _latent(h, W, m, eps):
    B, T = h.shape[:2]
    H, d, vd = m["heads"], m["dim"], m["vdim"]
    c = _rms(h @ W["dkv"].T, W["dkv.norm"], eps)
    o = _window_attend((h @ W["q"].T).reshape(B, T, H, d), (c @ W["uk"].T).reshape(B, T, H, d), (c @ W["uv"].T).reshape(B, T, H, vd), m["scale"],
                       (m.get("mask") or {}).get("size"), W["sink"])
    return (o * torch.sigmoid(h @ W["g"].T)[..., None]).reshape(B, T, -1) @ W["o"].T


def _mamba1(h, W, m, eps):
    n, r, N = m["inner"], m["dt_rank"], m["state"]
    xz = h @ W["in"].T
    x = torch.nn.functional.silu(_conv(xz[..., :n], W["conv"], W["conv.b"]))
    p = x @ W["x"].T
    dt = torch.nn.functional.softplus(p[..., :r] @ W["dt"].T + W["dt.b"])
    Bm, Cm, A = p[..., r:r + N], p[..., r + N:], -torch.exp(W["A_log"])
    s, y = torch.zeros((h.shape[0], n, N), dtype=F, device="cuda"), torch.empty_like(x)
    for t in range(h.shape[1]):
        s = torch.exp(dt[:, t, :, None] * A) * s + (dt[:, t] * x[:, t])[..., None] * Bm[:, t, None, :]
        y[:, t] = (s @ Cm[:, t, :, None])[..., 0]
    return ((y + W["D"] * x) * torch.nn.functional.silu(xz[..., n:])) @ W["o"].T


def _delta(h, W, m, eps):
    H, K, d, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    B, T = h.shape[:2]

    def part(name, heads, w):
        return torch.nn.functional.silu(_conv(h @ W[name].T, W[name + ".conv"])).reshape(B, T, heads, w)
    q, k, v = part("q", K, d), part("k", K, d), part("v", H, vd)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = (t.repeat_interleave(H // K, 2) for t in (q, k))
    beta = torch.sigmoid(h @ W["b"].T)
    a = ((h @ W["a1"].T) @ W["a2"].T + W["dt_bias"]).reshape(B, T, H, d)
    g = torch.exp(-torch.exp(W["A_log"])[:, None] * torch.nn.functional.softplus(a))
    gate = torch.sigmoid((h @ W["g1"].T) @ W["g2"].T).reshape(B, T, H, vd)
    s, o = torch.zeros((B, H, d, vd), dtype=F, device="cuda"), torch.empty_like(v)
    for t in range(T):
        s = g[:, t, :, :, None] * s
        u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ s)[..., 0, :])
        s = s + k[:, t, :, :, None] * u[:, :, None, :]
        o[:, t] = (q[:, t, :, None, :] @ s)[..., 0, :]
    return (_rms(o, W["norm"], eps) * gate).reshape(B, T, -1) @ W["o"].T


def _part(W, prefix):
    return {n[len(prefix):]: a for n, a in W.items() if n.startswith(prefix)}


def _fuzudra(W, cfg, toks):
    eps, D, T = cfg["norm"]["eps"], cfg["width"], toks.shape[1]
    ang = torch.arange(T, device="cuda", dtype=F)[:, None] * 10000.0 ** (-2.0 * torch.arange(D // 2, device="cuda", dtype=F) / D)
    x = W["embed"][toks] + torch.stack([torch.sin(ang), torch.cos(ang)], -1).reshape(T, D)
    mixers = {"latent_attention": _latent, "mamba1": _mamba1, "channel_delta": _delta}
    for i, L in enumerate(cfg["layers"]):
        P = _part(W, f"l{i}.")
        x = x + mixers[L["type"]](_rms(x, 1.0 + P["norm1"], eps), _part(P, "mix."), L["mixer"], eps)
        h = _rms(x, 1.0 + P["norm2"], eps)
        x = x + (torch.nn.functional.gelu(h @ P["mlp.gate"].T, approximate="tanh") * (h @ P["mlp.up"].T)) @ P["mlp.down"].T
    return _rms(x, 1.0 + W["final.norm"], eps)


def _layer_norm(x, w, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w


def _yarn(rot):
    n, base, s = rot["dims"], float(rot["base"]), rot["scaling"]
    i = np.arange(n // 2, dtype=np.float64)
    f = base ** (-2.0 * i / n)

    def at(turns):
        return n * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(at(s["fast"])), 0.0), min(math.ceil(at(s["slow"])), n - 1.0)
    ramp = np.clip((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return torch.from_numpy(f / s["factor"] * ramp + f * (1 - ramp)).cuda(), 0.1 * math.log(s["factor"]) + 1.0


def _musutar(W, cfg, toks):
    eps, B, T = cfg["norm"]["eps"], *toks.shape
    x = W["embed"][toks]
    xs = torch.stack([x] * cfg["streams"])
    kept = {}

    def turn(x, rot):
        f, m = _yarn(rot)
        a = torch.arange(T, device="cuda", dtype=F)[:, None, None] * f
        c, s = torch.cos(a) * m, torch.sin(a) * m
        u, v = x[..., :len(f)], x[..., len(f):2 * len(f)]
        return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * len(f):]], -1)

    def attention(h, P, m, i):
        H, G, d, vd = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        conv = lambda n, heads, w: _conv(h @ P[n].T, P[n + ".conv"]).reshape(B, T, heads, w)  # noqa: E731
        q = turn(conv("q", H, d), m["rot"])
        kept[i] = (turn(conv("k", G, d), m["rot"]), conv("v", G, vd)) if m.get("kv_from") is None else kept[m["kv_from"]]
        o = _window_attend(q, *kept[i], m["scale"], (m.get("mask") or {}).get("size"))
        return (o.reshape(B, T, -1) * torch.sigmoid(h @ P["g"].T)) @ P["o"].T

    def lightning(h, P, m, i):
        H, d, vd = m["heads"], m["dim"], m["vdim"]
        q, k, v = (torch.nn.functional.silu(h @ P[n].T).reshape(B, T, H, -1) for n in ("q", "k", "v"))
        decay = torch.tensor(m["decay"], dtype=F, device="cuda")[:, None, None]
        s, o = torch.zeros((B, H, d, vd), dtype=F, device="cuda"), torch.empty_like(v)
        for t in range(T):
            s = decay * s + k[:, t, :, :, None] * v[:, t, :, None, :]
            o[:, t] = (q[:, t, :, None, :] @ s)[..., 0, :]
        return (_rms(o.reshape(B, T, -1), P["norm"], eps) * torch.sigmoid(h @ P["g"].T)) @ P["o"].T

    for i, L in enumerate(cfg["layers"]):
        P = _part(W, f"l{i}.")
        for n in (1, 2):
            h = _layer_norm(torch.einsum("s,sbtd->btd", P[f"hc{n}.in"], xs), P[f"norm{n}"], eps)
            if n == 1:
                y = (attention if L["type"] == "attention" else lightning)(h + _conv(h, P["canon1"]), _part(P, "mix."), L["mixer"], i)
            else:
                y = torch.relu(h @ P["mlp.up"].T) ** 2 @ P["mlp.down"].T
            y = y * torch.sigmoid(h @ P[f"rg{n}"].T + P[f"rg{n}.b"])
            xs = torch.einsum("su,sbtd->ubtd", P[f"hc{n}.mix"], xs) + P[f"hc{n}.out"][:, None, None, None] * y[None]
    return _layer_norm(xs.sum(0), W["final.norm"], eps)


def _exact_accept(case, seed):
    p, q, draft, ua, us = (t.cpu() for t in _accept_inputs(case, seed))
    B, k = draft.shape
    n, tok = torch.zeros(B, dtype=torch.int32), torch.full((B, k + 1), -1, dtype=torch.int64)

    def soft(x):
        return torch.softmax(_kept(x / case["temperature"], case["top_k"]).to(F), -1)

    for b in range(B):
        i, rest = 0, None
        while i < k and rest is None:
            x, pi, qi = draft[b, i], soft(p[b, i]), soft(q[b, i])
            if float(ua[b, i]) * qi[x] < pi[x]:
                tok[b, i] = x
                i += 1
            else:
                rest = (pi - qi).clamp_min(0.0)
        rest = soft(p[b, k]) if rest is None else rest
        c = torch.cumsum(rest, 0)
        tok[b, i] = torch.searchsorted(c, c[-1] * float(us[b, i]), right=True)
        n[b] = i
    return {"len": n, "tokens": tok}


def exact(case, seed):
    kind = case["kind"]
    if kind == "accept":
        return _exact_accept(case, seed)
    if kind == "linear":
        x, w, b = (t.to(F) for t in _floats(case, seed))
        return x @ w.T + b
    if kind == "attention":
        q, k, v = (t.to(F) for t in _floats(case, seed))
        return torch.softmax(q @ k.transpose(1, 2) * case["dim"] ** -0.5, -1) @ v
    if kind == "verse":
        return _exact_verse(case, seed)
    cfg = _COMPOSED[kind][1](case["width"])
    W = {n: w.to(F) for n, w in _composed_weights(kind, cfg)}
    toks = torch.from_numpy(_tokens(case, seed)).cuda()
    hidden = (_fuzudra if kind == "fuzudra" else _musutar)(W, cfg, toks)
    if case["ctx"]:
        return hidden[:, case["ctx"]:] @ W["head"].T
    return torch.stack([hidden[b, n - 1] for b, n in enumerate(_lens(case))]) @ W["head"].T
