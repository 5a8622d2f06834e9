"""Quantised linears outside the split-K route: the tensor-core kernel against the mma.sync one on the same model, at row counts around its
blocks, one to three k groups, odd vocabularies and half groups."""

import numpy as np
import pytest

import versenext_b200 as vn
from oracle import model as OM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["int8", "int4", "int4g128"])
@pytest.mark.parametrize("dim,vocab,mod,B,T", [(128, 250, False, 1, 257), (64, 131, False, 3, 129), (192, 384, True, 2, 200), (512, 1000, False, 5, 111),
                                               (256, 256, True, 9, 64)])
def test_rows_kernel_equals_mma_sync(monkeypatch, scheme, dim, vocab, mod, B, T):
    cfg = OM.mate_config(vocab_size=vocab, dim=dim, n_layer=2, n_head=dim // 64, n_kv_head=1, window_size=40, num_global_tokens=8, max_seq_len=300, init_std=0.05,
                         num_dense_parts=2, num_experts_per_part=3, top_k=1, layer_pattern=["mod" if mod else "trisparse", "trisparse"])
    sd = {n: OM.bf16_round(v) for n, v in OM.init_state_dict(cfg, seed=3, gate_std=1.0).items()}
    kw = cfg.to_dict()
    kw.pop("init_std")
    toks = np.random.default_rng(0).integers(0, vocab, (B, T))
    got = []
    for old in (False, True):
        if old:
            monkeypatch.setenv("VN_GEMM_TCQ", "0")
        m = vn.VerseNexLM(dtype="bf16", **kw)
        m.load_state_dict(sd)
        m.quantize(scheme)
        cache = m.new_cache(B, T + 1)
        got.append(m.forward_cached(toks, cache).numpy())
        m.check()
    # the same products and scales in float32: only the order of the sums differs, and a bf16 rounding of it now and then
    assert np.linalg.norm(got[0] - got[1]) / np.linalg.norm(got[1]) < 4e-3


# every row count goes to the tensor-core kernel where a model is too wide for the split-K route: around its tiles of 16 and blocks of 128
# rows, a group and a half of inputs
@pytest.mark.parametrize("scheme", ["int8", "int4", "int4g128"])
@pytest.mark.parametrize("B,T", [(1, 1), (3, 5), (1, 17), (64, 2), (43, 3), (256, 1)])
def test_few_rows_of_a_wide_model(monkeypatch, scheme, B, T):
    cfg = OM.mate_config(vocab_size=131, dim=2112, n_layer=1, n_head=33, n_kv_head=3, window_size=40, num_global_tokens=8, max_seq_len=300, init_std=0.02,
                         layer_pattern=["trisparse"])
    sd = {n: OM.bf16_round(v) for n, v in OM.init_state_dict(cfg, seed=3, gate_std=1.0).items()}
    kw = cfg.to_dict()
    kw.pop("init_std")
    toks = np.random.default_rng(0).integers(0, 131, (B, 7 + T))
    got = []
    for old in (False, True):
        if old:
            monkeypatch.setenv("VN_GEMM_TCQ", "0")
        m = vn.VerseNexLM(dtype="bf16", **kw)
        m.load_state_dict(sd)
        m.quantize(scheme)
        cache = m.new_cache(B, T + 8)
        m.forward_cached(toks[:, :7], cache, want_logits=False, want_hidden=True, last_only=True)
        cache.commit(7, np.full(B, 7, np.int32))
        got.append(m.forward_cached(toks[:, 7:], cache).numpy())
        m.check()
    assert np.linalg.norm(got[0] - got[1]) / np.linalg.norm(got[1]) < 4e-3     # as above


@pytest.mark.parametrize("mod", [False, True])
def test_switch_of_a_prompts_gemms(monkeypatch, mod):
    """VN_PREFILL_TC=0 keeps a prompt's GEMMs on mma.sync, quantised or not; the last rows' head has few rows."""
    from test_prompt_pairs_gpu import _kernels
    cfg = OM.mate_config(vocab_size=131, dim=128, n_layer=1, n_head=2, n_kv_head=1, window_size=40, num_global_tokens=8, max_seq_len=300, init_std=0.05,
                         num_dense_parts=2, num_experts_per_part=3, top_k=1, layer_pattern=["mod" if mod else "trisparse"])
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype="bf16", **kw)
    m.load_state_dict(OM.init_state_dict(cfg, seed=3))
    m.quantize("int8")
    toks = m.ctx.from_numpy(np.random.default_rng(0).integers(0, 131, (3, 100)))
    for flag in ("1", "0"):
        monkeypatch.setenv("VN_PREFILL_TC", flag)
        _, names = _kernels(lambda: m.forward_cached(toks, m.new_cache(3, 101)))
        assert any("gemm_tcq_rows_kernel" in n for n in names) == (flag == "1"), names
        assert any("gemm_mma_q_kernel" in n for n in names) == (flag == "0"), names
