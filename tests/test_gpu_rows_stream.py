"""Products of one token, and of five to thirty-one, with bf16 weights (four columns per warp, slices of K over warps): columns that do not fill a warp's four, lengths around a lane's
pieces and around the slices, every epilogue that pairs columns, the chosen experts' products."""
import numpy as np
import pytest

from xalm_b200 import capi

pytestmark = pytest.mark.gpu


def bf16(a):
    return (np.ascontiguousarray(a, np.float32).view(np.uint32) + 0x8000 & 0xFFFF0000).view(np.float32)


def bound(K):
    """fp32 sums of K products of order K^-1/2 in K / 256 steps per lane and a tree: far below sqrt(K) roundings of values of order one."""
    return 2.0 ** -23 * (K ** 0.5 + 8) * 4


@pytest.mark.parametrize("N", [1, 2, 3, 4, 7, 33, 2500])
@pytest.mark.parametrize("K", [8, 248, 256, 264, 512, 1000, 2048, 4104])
@pytest.mark.parametrize("T", [1, 5, 8, 9, 16, 17, 31])
def test_plain_and_paired_columns(N, K, T):
    rng = np.random.default_rng(N * K)
    x, w, u = rng.standard_normal((T, K)).astype(np.float32), bf16(rng.standard_normal((N, K)) / K ** 0.5), bf16(rng.standard_normal((N, K)) / K ** 0.5)
    z, y = x.astype(np.float64) @ w.T, x.astype(np.float64) @ u.T
    mul = rng.standard_normal((T, N)).astype(np.float32)
    got = capi.rows_act(x, w, act=0, cap=20.0, mul=mul, w_bf16=True)
    assert np.abs(got - 20 * np.tanh(z / 20) / (1 + np.exp(-mul))).max() < bound(K)
    got = capi.glu_rows(x, w, u, 7.0, w_bf16=True)
    g = np.minimum(z, 7.0)
    assert np.abs(got - g / (1 + np.exp(-1.702 * g)) * (np.clip(y, -7, 7) + 1)).max() < 4 * bound(K)


@pytest.mark.parametrize("T,K,ff", [(1, 64, 24), (1, 1032, 40), (3, 256, 6), (2, 2048, 130), (17, 256, 6), (31, 1032, 130), (20, 64, 24)])
def test_chosen_experts(T, K, ff):
    rng = np.random.default_rng(K + ff)
    E, top = 6, 2
    h = rng.standard_normal((T, K)).astype(np.float32)
    wr = bf16(rng.standard_normal((E, K)) * 3 / K ** 0.5)
    wg, wu, wd = (bf16(rng.standard_normal(s) / s[2] ** 0.5) for s in ((E, ff, K), (E, ff, K), (E, K, ff)))
    idx, wgt, out = capi.moe_ffn(h, wr, wg, wu, wd, top, w_bf16=True)
    for t in range(T):
        for r in range(top):
            e, x = idx[t, r], h[t].astype(np.float64)
            g = wg[e].astype(np.float64) @ x
            want = wd[e].astype(np.float64) @ (g / (1 + np.exp(-g)) * (wu[e].astype(np.float64) @ x))
            assert np.abs(out[t, r] - want).max() < 4 * bound(K) + 4 * bound(ff)


@pytest.mark.parametrize("W,groups", [(64, 1), (96, 3), (1024, 8), (4096, 1), (4096, 8), (8192, 1)])
@pytest.mark.parametrize("T", [1, 4])
def test_group_norm_of_short_steps(W, groups, T):
    rng = np.random.default_rng(W + groups)
    parts, n_hist = 3, 5
    y, pw, w, x = rng.standard_normal((T, parts, W)), rng.uniform(0.1, 1, (T, parts)), 1 + 0.2 * rng.standard_normal(W), rng.standard_normal((T, W))
    hist, coef = rng.standard_normal((n_hist, T, W)), rng.standard_normal(n_hist + 1)
    u = (y * pw[:, :, None]).sum(1).reshape(T, groups, -1)
    want = x + (u / np.sqrt((u * u).mean(-1, keepdims=True) + 1e-5)).reshape(T, W) * w
    got, avg = capi.group_norm_residual(y, w, groups, 1e-5, x_in=x, part_w=pw, hist=hist, dwa=coef)
    assert np.abs(got - want).max() < 2e-5  # a dozen fp32 roundings of values below 8
    assert np.abs(avg - ((coef[:-1, None, None] * hist).sum(0) + coef[-1] * want)).max() < 6e-5


@pytest.mark.parametrize("N", [1000, 4720, 4721, 9001])
@pytest.mark.parametrize("K", [1, 9, 511, 1030])
def test_one_token_of_rows_that_are_not_whole_pieces(N, K):
    """K in slices below 4721 columns (from 512 on); the one-token instance for the others."""
    rng = np.random.default_rng(N + K)
    x, w = rng.standard_normal((1, K)).astype(np.float32), bf16(rng.standard_normal((N, K)) / K ** 0.5)
    got = capi.rows_act(x, w, act=0, w_bf16=True)
    z = x.astype(np.float64) @ w.T
    assert np.abs(got - z).max() < 2 * bound(K)
