"""Prompts whose GEMMs run on SM pairs against the mma.sync kernels on the same model: odd features (half a tile, a pair whose second CTA
has none), rows that do not fill a segment, experts' pieces of every length; which products the pairs take, with the functions,
biases and partial k blocks that composed models bring."""

import numpy as np
import pytest

import versenext_b200 as vn
from oracle import model as OM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,vocab,mod,B,T,every", [(512, 1000, False, 7, 443, False), (320, 900, False, 13, 300, True), (128, 38000, False, 1, 390, True),
                                                     (256, 77, True, 31, 167, False), (1024, 300, True, 2, 1025, False)])
def test_pair_kernel_equals_mma_sync(monkeypatch, dim, vocab, mod, B, T, every):
    cfg = OM.mate_config(vocab_size=vocab, dim=dim, n_layer=2, n_head=dim // 64, n_kv_head=1, window_size=60, num_global_tokens=8, max_seq_len=1100, init_std=0.04,
                         num_dense_parts=2, num_experts_per_part=5, top_k=2, layer_pattern=["mod" if mod else "trisparse", "trisparse"])
    sd = {n: OM.bf16_round(v) for n, v in OM.init_state_dict(cfg, seed=3, gate_std=1.0).items()}
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype="bf16", **kw)
    m.load_state_dict(sd)
    toks = np.random.default_rng(0).integers(0, vocab, (B, T))
    got = []
    for tc in ("1", "0"):
        monkeypatch.setenv("VN_PREFILL_TC", tc)
        cache = m.new_cache(B, T + 1)
        got.append(m.forward_cached(toks, cache, want_logits=every, want_hidden=not every).numpy())
        m.check()
    # products of the same bf16 operands with float32 sums: another order, and a bf16 rounding of it now and then
    assert np.linalg.norm(got[0] - got[1]) / np.linalg.norm(got[1]) < 6e-3


def _kernels(f):
    """(result of f, names of the kernels that ran in it)"""
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = f()
        torch.cuda.synchronize()
    return out, {e.key for e in prof.key_averages()}


def _pairs(names, mode):
    """Whether the SM-pair kernel ran with an epilogue: 1 stores, 2 gated pairs, 3 residual adds."""
    return any(f"gemm_tc2_kernel<{mode}>" in n for n in names)


def _verse(dim, vocab):
    cfg = OM.mate_config(vocab_size=vocab, dim=dim, n_layer=1, n_head=dim // 64, n_kv_head=1, window_size=60, num_global_tokens=8, max_seq_len=1100, init_std=0.04,
                         layer_pattern=["trisparse"])
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype="bf16", **kw)
    m.load_state_dict({n: OM.bf16_round(v) for n, v in OM.init_state_dict(cfg, seed=3, gate_std=1.0).items()})
    return m


# (what the SM pairs take: 1 stores = the head here, 2 gated pairs, 3 residual adds.)  A vocabulary whose last tile leaves the second CTA
# without features, with segments of an odd number of chunks; few rows; short K; widths that fill tiles badly
@pytest.mark.parametrize("dim,vocab,B,T,modes", [(512, 38000, 1, 672, {1}), (512, 1000, 8, 512, {2, 3}), (1024, 8200, 5, 500, {1, 2, 3}), (512, 38000, 1, 300, set()),
                                                 (128, 38000, 4, 512, set()), (320, 600, 3, 512, set()), (320, 600, 4, 512, {3})])
def test_which_products_run_on_pairs(monkeypatch, dim, vocab, B, T, modes):
    m = _verse(dim, vocab)
    toks = m.ctx.from_numpy(np.random.default_rng(0).integers(0, vocab, (B, T)))
    got = []
    for tc in ("1", "0"):
        monkeypatch.setenv("VN_PREFILL_TC", tc)
        cache = m.new_cache(B, T + 1)
        out, names = _kernels(lambda: m.forward_cached(toks, cache))
        assert {k for k in (1, 2, 3) if _pairs(names, k)} == (modes if tc == "1" else set()), names
        got.append(out.numpy())
        m.check()
    assert np.linalg.norm(got[0] - got[1]) / np.linalg.norm(got[1]) < 6e-3     # as above


def _composed(cases, layers, B, n, monkeypatch, modes, **config):
    cfg = cases.config(layers, vocab=90, **config)
    m = cases.build(cfg, cases.weights(cfg, seed=4), "bf16")
    toks, got = np.random.default_rng(2).integers(0, 90, B * n), []
    for tc in ("1", "0"):
        monkeypatch.setenv("VN_PREFILL_TC", tc)
        cache = m.new_cache(B, n + 1)
        out, names = _kernels(lambda: m.forward_ragged(cache, np.arange(B, dtype=np.int32), np.full(B, n, np.int32), toks, np.arange(0, B * n, 37)))
        if tc == "1":
            assert {k for k in (1, 2, 3) if _pairs(names, k)} == modes, names
        got.append(out.numpy())
        m.check()
    return np.linalg.norm(got[0] - got[1]) / np.linalg.norm(got[1])


def test_functions_and_16_bit_results_on_pairs(monkeypatch):
    """Dense 16-bit results, silu on some columns of a product and the squared ReLU: a linear attention layer with a plain feed-forward."""
    import musutar_cases as C
    assert _composed(C, [C.lightning(heads=20, dim=64, vdim=64, ff=4096)], 5, 520, monkeypatch, {1}, width=1024) < 2e-2   # a layer's 16-bit roundings


def test_biases_on_pairs(monkeypatch):
    """Residual adds with a bias."""
    import bozasun_cases as C
    assert _composed(C, [C.attention(heads=16, kv_heads=4, dim=64, vdim=64, rot=32, mlp=C.dense(1536))], 3, 500, monkeypatch, {3}, width=1024) < 2e-2


def test_half_k_blocks_on_pairs(monkeypatch):
    """Experts whose inputs end inside a block of k."""
    import bozasun_cases as C
    mlp = C.moe(experts=7, identity=3, top=3, groups=5, keep=2, ff=1024)
    assert _composed(C, [C.attention(mlp=mlp)], 5, 520, monkeypatch, {2}, width=264) < 2e-2


def test_clamped_experts_on_pairs(monkeypatch):
    """The clamped gated function on pairs, experts' inputs weighed first."""
    import givozen_cases as C
    mlp = C.moe(experts=7, top=3, ff=1024, shared_ff=64)
    assert _composed(C, [C.attention(mlp=mlp)], 5, 520, monkeypatch, {2}, width=264) < 2e-2
