"""Prompts long enough for the SM-pair GEMM against the mma.sync kernels on the same model: odd features (half a tile, a pair whose
second CTA has none), rows that do not fill a segment, K that does not fill a block, and experts' pieces of every length."""

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
