"""fp32 operators at the sizes where their kernels change or end: tile remainders, rows that start off 16 bytes, few rows,
wide heads; against float64, within the bound of a float32 sum in any order."""

import numpy as np
import pytest

import versenext_b200 as vn

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -24


@pytest.mark.parametrize("M,N,K", [(1, 1, 4), (1, 1030, 128), (2, 5, 64), (3, 4099, 132), (7, 66, 176), (16, 63, 68), (17, 257, 20), (32, 1025, 256),
                                   (33, 65, 33), (63, 127, 16), (64, 128, 15), (65, 129, 17), (5, 130, 31), (500, 1000, 100), (1000, 2752, 36), (70, 64, 1)])
@pytest.mark.parametrize("op", ["linear", "matmul"])
def test_products(op, M, N, K):
    rng = np.random.default_rng(M * 7919 + N * 31 + K)
    x, w, b = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), (N, K), (N,)))
    be = vn.get_backend("cuda")
    got = be.linear(x, w, b).numpy() if op == "linear" else be.matmul(x, np.ascontiguousarray(w.T)).numpy()
    x, w, b = (a.astype(np.float64) for a in (x, w, b if op == "linear" else 0 * b))
    bound = (K + 2) * EPS * (np.abs(x) @ np.abs(w).T + np.abs(b)) * 1.01
    assert np.all(np.abs(got - (x @ w.T + b)) <= bound)


@pytest.mark.parametrize("BH,Tq,Tk,D", [(1, 1, 1, 1), (3, 1, 77, 64), (2, 15, 500, 48), (2, 16, 16, 32), (1, 64, 64, 64), (3, 65, 63, 30), (2, 33, 129, 128),
                                        (2, 130, 65, 100), (1, 20, 70, 33), (1, 17, 40, 200), (2, 1, 3000, 20)])
@pytest.mark.parametrize("masked", [False, True])
def test_attention(BH, Tq, Tk, D, masked):
    rng = np.random.default_rng(BH * 7919 + Tq * 31 + Tk + D)
    q, k, v = (rng.standard_normal((BH, n, D)).astype(np.float32) for n in (Tq, Tk, Tk))
    mask = np.where(rng.random((Tq, Tk)) < 0.3, -np.inf, rng.standard_normal((Tq, Tk))).astype(np.float32) if masked else None
    if masked:
        mask[0] = np.finfo(np.float32).min                 # a row with nothing but the lowest value: all keys alike
        mask[1:, 0] = 0.0
        mask[-1, :] = -np.inf if Tq > 1 else mask[-1]      # and one with nothing at all
    got = vn.get_backend("cuda").attention(q, k, v, mask).numpy()
    s = q.astype(np.float64) @ k.astype(np.float64).transpose(0, 2, 1) / np.sqrt(D)
    # scores in float32: a dot product of D terms, the scale and the mask, then exponentials and sums over Tk
    err = (D + 4) * EPS * (np.abs(q) @ np.abs(k).transpose(0, 2, 1)).max() / np.sqrt(D) + 8 * EPS
    if masked:
        s = s + mask.astype(np.float64)
        s[:, 0] = 0.0                                      # float32 absorbs the scores into the lowest value
        err += 8 * EPS * np.abs(np.where(np.isfinite(mask) & (mask > -1e30), mask, 0)).max()
    with np.errstate(invalid="ignore"):
        p = np.exp(s - s.max(-1, keepdims=True))
        want = (p / p.sum(-1, keepdims=True)) @ v.astype(np.float64)
    if masked and Tq > 1:
        assert np.all(np.isnan(got[:, -1])) and np.all(np.isnan(want[:, -1]))
        got, want = got[:, :-1], want[:, :-1]
    assert np.all(np.abs(got - want) <= (2 * err + (Tk + 8) * EPS) * np.abs(v).max())


@pytest.mark.parametrize("n_head,n_kv,dim,window,n_sink,alibi,ctx,new,tree", [
    (4, 4, 64, 32, 4, True, 40, 5, False), (4, 2, 96, 16, 3, True, 0, 70, False), (2, 1, 128, 24, 1, False, 70, 1, False), (4, 1, 160, 64, 65, True, 61, 17, False),
    (8, 2, 64, 1100, 2, True, 1020, 3, False), (8, 2, 64, 100, 2, True, 1023, 3, False), (4, 2, 256, 20, 7, True, 30, 9, True), (2, 2, 32, 8, 1, False, 0, 400, False)])
def test_three_path_attention(n_head, n_kv, dim, window, n_sink, alibi, ctx, new, tree):
    """Rows of the float32 model's attention at the edges of its blocks (rows that do not fill one, groups of query heads,
    contexts around a key tile, the window, ALiBi's switch, more blocks than SMs) against the restated forward."""
    from oracle import model as OM
    cfg = OM.small_config(vocab_size=50, dim=dim, n_layer=1, n_head=n_head, n_kv_head=n_kv, window_size=window, num_global_tokens=n_sink,
                          use_alibi=alibi, use_rope=not alibi, max_seq_len=2048, init_std=0.2)
    sd = OM.init_state_dict(cfg, seed=5, gate_std=1.0)
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype="f32", **kw)
    m.load_state_dict(sd)
    B = 40 if new >= 400 else 2
    toks = np.random.default_rng(1).integers(0, 50, (B, ctx + new))
    parents = [-1, -1, 0, 0, 1, 2, 2, 5, 4][:new] if tree else None
    cache, oc = m.new_cache(B, ctx + new + 1), None
    if ctx:
        m.forward_cached(toks[:, :ctx], cache, last_only=True)
        cache.commit(ctx, np.full(B, ctx, np.int32))
        _, oc = OM.forward(sd, cfg, toks[:, :ctx])
    got = m.forward_cached(toks[:, ctx:], cache, parents=parents).numpy()
    want, _ = OM.forward(sd, cfg, toks[:, ctx:], cache=oc, parents=parents)
    assert np.max(np.abs(got - want)) / np.max(np.abs(want)) < 1e-4      # float32 on both sides, sums in other orders


@pytest.mark.parametrize("n_head,n_kv,dim,window,B,T", [(4, 4, 64, 8, 1, 40), (4, 2, 256, 5, 2, 300), (2, 1, 32, 3, 40, 12)])
def test_a_value_that_is_no_number_stays_in_its_window(n_head, n_kv, dim, window, B, T):
    """A token whose embedding is NaN puts NaN into the keys and values of its position.  Rows whose window ends before it are what they
    are with any other token there, although their block's neighbours see the position."""
    from oracle import model as OM
    cfg = OM.small_config(vocab_size=50, dim=dim, n_layer=1, n_head=n_head, n_kv_head=n_kv, window_size=window, num_global_tokens=2,
                          use_alibi=False, use_rope=True, max_seq_len=512, init_std=0.2)
    sd = OM.init_state_dict(cfg, seed=5, gate_std=1.0)
    sd["tok_emb.weight"] = sd["head.weight"] = sd["tok_emb.weight"].copy()
    sd["tok_emb.weight"][49] = np.nan
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype="f32", **kw)
    m.load_state_dict(sd)
    toks = np.random.default_rng(1).integers(0, 49, (B, T))
    got = []
    for first in (7, 49):
        toks[:, 0] = first
        got.append(m.forward_cached(toks, m.new_cache(B, T), want_logits=False, want_hidden=True).numpy())
    assert np.all(np.isnan(got[1][:, :window])) and np.all(np.isfinite(got[0]))
    np.testing.assert_array_equal(got[0][:, window:], got[1][:, window:])


def test_threads_launch_two_sizes():
    """One context per thread: the shared memory that a kernel may ask for belongs to the function, so a smaller launch of one thread must
    not take away what a larger one of the other is about to use."""
    import threading
    be, rng, results = vn.get_backend("cuda"), np.random.default_rng(3), {}

    def run(Tk, q, k, v):
        ctx = vn.Context(0)
        try:
            d = [ctx.from_numpy(a) for a in (q, k, v)]
            out = ctx.empty(q.shape, np.float32)
            for _ in range(4000):
                ctx._check(ctx.lib.vn_attention(ctx.handle, *(a.ptr for a in d), None, out.ptr, 1, 2, Tk, 4))
            results[Tk] = out.numpy()
        except RuntimeError as e:
            results[Tk] = e

    inputs = {Tk: [rng.standard_normal((1, n, 4)).astype(np.float32) for n in (2, Tk, Tk)] for Tk in (12800, 12100)}
    threads = [threading.Thread(target=run, args=(Tk, *a)) for Tk, a in inputs.items()]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for Tk, a in inputs.items():
        assert not isinstance(results[Tk], Exception), results[Tk]
        np.testing.assert_array_equal(results[Tk], be.attention(*a).numpy())


@pytest.mark.parametrize("Tq,D", [(2, 8), (2, 200), (20, 30), (70, 64), (65, 128)])
def test_attention_of_values_near_the_largest(Tq, D):
    """A weighted mean is no larger than what it is taken of: values of 3e38 over hundreds of keys stay finite."""
    rng = np.random.default_rng(Tq + D)
    q, k = (rng.standard_normal((2, n, D)).astype(np.float32) for n in (Tq, 500))
    v = (3e38 * np.sign(rng.standard_normal(D)) * np.ones((2, 500, D))).astype(np.float32)
    got = vn.get_backend("cuda").attention(q, k, v).numpy().astype(np.float64)
    assert np.all(np.abs(got / v[:, :1].astype(np.float64) - 1) <= (500 + 8 * 8 + 8) * EPS)   # 500 weights, eight tiles' rescaling


# window and cache of thousands of keys, short contexts (the kernel is chosen by what a block may see): few blocks of one SM each, blocks that
# share SMs, more blocks than the SMs hold at once, scores beyond shared memory
@pytest.mark.parametrize("window,B,T,ctx,kernel", [(9000, 1, 5, 30, "rows"), (9000, 2, 200, 0, "attn"), (10000, 1, 5, 30, "attn"), (10000, 2, 40, 7, "attn"),
                                                   (4000, 2, 200, 0, "rows"), (6000, 2, 200, 3, "attn"), (3000, 8, 100, 0, "rows"), (40, 64, 5, 9, "rows")])
@pytest.mark.parametrize("alibi", [False, True])
def test_wide_windows(window, B, T, ctx, kernel, alibi):
    from oracle import model as OM
    cfg = OM.small_config(vocab_size=50, dim=64, n_layer=1, n_head=4, n_kv_head=2, window_size=window, num_global_tokens=3, use_alibi=alibi,
                          use_rope=not alibi, max_seq_len=window + 100, init_std=0.2)
    sd = OM.init_state_dict(cfg, seed=5, gate_std=1.0)
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype="f32", **kw)
    m.load_state_dict(sd)
    toks = np.random.default_rng(1).integers(0, 50, (B, ctx + T))
    cache, oc = m.new_cache(B, window + 100), None
    if ctx:
        m.forward_cached(toks[:, :ctx], cache, last_only=True)
        cache.commit(ctx, np.full(B, ctx, np.int32))
        _, oc = OM.forward(sd, cfg, toks[:, :ctx])
    m.ctx.profile(True)
    got = m.forward_cached(toks[:, ctx:], cache).numpy()
    ran = m.ctx.profile_report()
    m.ctx.profile(False)
    assert any(f"trisparse_{kernel}_kernel" in name for name in ran), list(ran)
    want, _ = OM.forward(sd, cfg, toks[:, ctx:], cache=oc)
    assert np.max(np.abs(got - want)) / np.max(np.abs(want)) < 1e-4      # float32 on both sides, sums in other orders


# few keys: a block or a warp per row, on both sides of 512 rows, of a warp's lanes and of eight rows a block
@pytest.mark.parametrize("BH,Tq,Tk,D", [(1, 600, 1, 1), (2, 300, 8, 33), (3, 200, 32, 16), (5, 128, 16, 32), (600, 1, 8, 100), (1, 513, 5, 128), (64, 8, 32, 64),
                                        (2, 16, 32, 128), (1, 512, 31, 30), (103, 5, 7, 3)])
@pytest.mark.parametrize("masked", [False, True])
def test_attention_of_few_keys(BH, Tq, Tk, D, masked):
    test_attention(BH, Tq, Tk, D, masked)


# matrices of many features: every number of rows that a pass takes, passes that are not full
@pytest.mark.parametrize("M,N,K", [(1, 20001, 132), (2, 18944, 64), (3, 19003, 4), (4, 18945, 128), (7, 20011, 36), (8, 18950, 260), (17, 18947, 68), (32, 19001, 128)])
def test_linears_of_many_features(M, N, K):
    test_products("linear", M, N, K)


def test_wide_windows_of_many_rows():
    """More rows than the one-warp kernel's grid has: the rows kernel, whatever is faster.  Every sequence alike, so that one is the answer."""
    from oracle import model as OM
    cfg = OM.small_config(vocab_size=50, dim=32, n_layer=1, n_head=1, n_kv_head=1, window_size=6000, num_global_tokens=3, use_alibi=False, use_rope=True,
                          max_seq_len=6100, init_std=0.2)
    sd = OM.init_state_dict(cfg, seed=5, gate_std=1.0)
    kw = cfg.to_dict()
    kw.pop("init_std")
    m = vn.VerseNexLM(dtype="f32", **kw)
    m.load_state_dict(sd)
    toks = np.random.default_rng(1).integers(0, 50, (1, 50))
    got = m.forward_cached(np.repeat(toks, 1400, 0), m.new_cache(1400, 6050), want_logits=False, want_hidden=True).numpy()
    want, _ = OM.forward_hidden(sd, cfg, toks)
    assert np.max(np.abs(got - want)) / np.max(np.abs(want)) < 1e-4
