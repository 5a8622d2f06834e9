"""The gated function and the RMSNorm of the model kernels, on models whose attention and feed-forward add nothing: the hidden rows are
then the norms of the embedded tokens, value by value."""

import numpy as np
import pytest

import versenext_b200 as vn
from oracle import model as OM

pytestmark = pytest.mark.gpu
F32 = np.float32


def _model(sd, cfg, dtype, quant=None):
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype=dtype, **kw)
    m.load_state_dict(sd)
    if quant:
        m.quantize(quant)
    return m


def _weights(cfg, seed):
    sd = {n: OM.bf16_round(v) for n, v in OM.init_state_dict(cfg, seed=seed).items()}
    for n in sd:
        if n.endswith("attn.proj.weight"):
            sd[n] = np.zeros_like(sd[n])
    return sd


# one token, a verification block and a prompt; whole tiles of the prompt kernels on one SM and on SM pairs; quantised weights
@pytest.mark.parametrize("dim,B,T,quant", [(128, 1, 1, None), (1024, 2, 5, None), (128, 2, 150, None), (512, 8, 512, None), (128, 3, 100, "int8"), (128, 2, 3, "int8")])
def test_closed_gates_add_nothing(dim, B, T, quant):
    """silu as the reference computes it, x * 0.5 * (1 + tanh(x / 2)) in float32 (verse_torch/tensor.py:853-856), is zero from x = -19 down.
    With gates of -21 and below, ups of 1e8 leave the residual stream as it was, in every kernel that applies the function."""
    cfg = OM.small_config(vocab_size=64, dim=dim, n_layer=1, n_head=dim // 64, n_kv_head=1, max_seq_len=600, init_std=0.5)
    sd = _weights(cfg, 3)
    emb, p = sd["tok_emb.weight"].copy(), "blocks.0.ffn."
    emb[:, 0] = 8.0
    sd["tok_emb.weight"] = sd["head.weight"] = emb
    first = np.min(emb[:, 0] / np.sqrt(np.mean(emb * emb, -1)))               # of the normalised rows
    sd[p + "w_gate.weight"] = np.zeros_like(sd[p + "w_gate.weight"])
    sd[p + "w_up.weight"] = np.zeros_like(sd[p + "w_up.weight"])
    sd[p + "w_gate.weight"][:, 0] = OM.bf16_round(np.full(1, -22.0 / first, F32))
    sd[p + "w_up.weight"][:, 0] = OM.bf16_round(np.full(1, 1e8, F32))
    m = _model(sd, cfg, "bf16", quant)
    toks = np.random.default_rng(0).integers(0, 64, (B, T))
    got = m.forward_cached(toks, m.new_cache(B, T + 1), want_logits=False, want_hidden=True).numpy()
    m.check()
    want = OM.rmsnorm(emb[toks], np.ones(dim, F32))
    assert np.max(np.abs(got - want)) <= 8 * 2.0 ** -24 * np.max(np.abs(want)) + dim * 2.0 ** -24


# heads of 8; a row that does not fill its threads, one that does, one of many values a thread, one that is read twice
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("dim,B,T", [(72, 1, 3), (256, 2, 40), (1024, 1, 65), (1032, 1, 300), (4096, 1, 9), (4160, 1, 5)])
def test_norm_keeps_the_order_of_its_sum(dtype, dim, B, T):
    """A row's squares are added by 256 threads, thread t taking t, t + 256, ..., then lane by lane and warp by warp."""
    cfg = OM.small_config(vocab_size=64, dim=dim, n_layer=1, n_head=dim // 8, n_kv_head=1, max_seq_len=600, init_std=0.5)
    sd = _weights(cfg, 4)
    rng = np.random.default_rng(1)
    sd["blocks.0.ffn.w_down.weight"] = np.zeros_like(sd["blocks.0.ffn.w_down.weight"])
    sd["norm.weight"] = OM.bf16_round(rng.standard_normal(dim).astype(F32))
    m = _model(sd, cfg, dtype)
    toks = rng.integers(0, 64, (B, T))
    got = m.forward_cached(toks, m.new_cache(B, T + 1), want_logits=False, want_hidden=True).numpy()
    x = sd["tok_emb.weight"][toks].reshape(-1, dim).astype(F32)
    pad = np.zeros((len(x), -(-dim // 256) * 256), F32)
    pad[:, :dim] = x
    s = np.zeros((len(x), 256), F32)
    for part in pad.reshape(len(x), -1, 256).transpose(1, 0, 2).astype(np.float64):
        s = (part * part + s).astype(F32)                                     # a fused multiply-add: 16-bit squares, one rounding
    s = s.reshape(len(x), 8, 32)
    for o in (16, 8, 4, 2, 1):
        s = s + s[:, :, np.arange(32) ^ o]
    tot = np.zeros(len(x), F32)
    for w in range(8):
        tot = tot + s[:, w, 0]
    r = np.sqrt(tot / F32(dim) + F32(1e-6)).astype(F32)[:, None]
    assert np.array_equal(got.reshape(-1, dim), x / r * sd["norm.weight"])
