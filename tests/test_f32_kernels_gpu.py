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
