"""Products of 32 and more tokens with bf16 weights that stay in fp32 grade (rows_mma_kernel): sizes around its 64 x 64 tiles and 32-channel steps, every
epilogue that pairs columns, and what is not finite against the fp32 FMA tiles."""
import numpy as np
import pytest

from xalm_b200 import capi

pytestmark = pytest.mark.gpu


def bf16(a):
    return (np.ascontiguousarray(a, np.float32).view(np.uint32) + 0x8000 & 0xFFFF0000).view(np.float32)


def bound(K):
    """Exact products of order K^-1/2; K / 16 sums in fp32, each truncated or rounded: far below sqrt(K) roundings of values of order one."""
    return 2.0 ** -23 * (K ** 0.5 + 8) * 4


@pytest.mark.parametrize("N", [1, 2, 31, 63, 64, 65, 130])
@pytest.mark.parametrize("K", [8, 24, 32, 40, 256, 1000])
@pytest.mark.parametrize("T", [32, 63, 64, 65, 200])
def test_plain_and_paired_columns(T, K, N):
    rng = np.random.default_rng(N * K + T)
    x, w, u = rng.standard_normal((T, K)).astype(np.float32), bf16(rng.standard_normal((N, K)) / K ** 0.5), bf16(rng.standard_normal((N, K)) / K ** 0.5)
    z, y = x.astype(np.float64) @ w.T, x.astype(np.float64) @ u.T
    mul = rng.standard_normal((T, N)).astype(np.float32)
    got = capi.rows_act(x, w, act=0, cap=20.0, mul=mul, w_bf16=True)
    assert np.abs(got - 20 * np.tanh(z / 20) / (1 + np.exp(-mul))).max() < bound(K)
    got = capi.glu_rows(x, w, u, 7.0, w_bf16=True)
    g = np.minimum(z, 7.0)
    assert np.abs(got - g / (1 + np.exp(-1.702 * g)) * (np.clip(y, -7, 7) + 1)).max() < 4 * bound(K)


@pytest.mark.parametrize("val", [np.inf, -np.inf, np.nan, 3.4e38])
def test_what_is_not_finite_stays_with_its_row(val):
    rng = np.random.default_rng(3)
    x, w = rng.standard_normal((70, 96)).astype(np.float32), bf16(rng.standard_normal((80, 96)))
    x[40, 33] = val
    got, want = capi.rows_act(x, w, act=0, w_bf16=True), capi.rows_act(x, w, act=0, w_bf16=False)
    for f in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(f(got), f(want))
    rows = np.arange(70) != 40
    assert np.abs(got[rows] - want[rows]).max() < 2e-4  # sums of 96 products of order one, in another order


# 64 x 64 outputs per CTA: from 148 tiles on, or one step of channels.  Steps of whole and part rounds; two columns a store and one
@pytest.mark.parametrize("T,N", [(700, 1000), (640, 961)])
@pytest.mark.parametrize("K", [40, 64, 256, 1000])
def test_many_tiles(T, N, K):
    rng = np.random.default_rng(N + K)
    x, w, u = rng.standard_normal((T, K)).astype(np.float32), bf16(rng.standard_normal((N, K)) / K ** 0.5), bf16(rng.standard_normal((N, K)) / K ** 0.5)
    z, y = x.astype(np.float64) @ w.T, x.astype(np.float64) @ u.T
    assert np.abs(capi.rows_act(x, w, act=0, w_bf16=True) - z).max() < bound(K)                     # plain rows
    mul = rng.standard_normal((T, N)).astype(np.float32)
    assert np.abs(capi.rows_act(x, w, act=0, cap=20.0, mul=mul, w_bf16=True) - 20 * np.tanh(z / 20) / (1 + np.exp(-mul))).max() < bound(K)
    g = np.minimum(z, 7.0)
    assert np.abs(capi.glu_rows(x, w, u, 7.0, w_bf16=True) - g / (1 + np.exp(-1.702 * g)) * (np.clip(y, -7, 7) + 1)).max() < 4 * bound(K)


@pytest.mark.parametrize("val", [np.inf, -np.inf, np.nan, 3.4e38])
def test_what_is_not_finite_in_many_tiles(val):
    rng = np.random.default_rng(4)
    x, w = rng.standard_normal((700, 96)).astype(np.float32), bf16(rng.standard_normal((960, 96)))
    x[640, 70] = val                                                                                # (the last step of three)
    got, want = capi.rows_act(x, w, act=0, w_bf16=True), capi.rows_act(x, w, act=0, w_bf16=False)
    for f in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(f(got), f(want))
    rows = np.arange(700) != 640
    assert np.abs(got[rows] - want[rows]).max() < 2e-4                                              # as above


# per-head products of a latent (batches whose rows, weights, outputs and gates advance): 32 x 32 outputs a CTA in both, in the second, in neither
@pytest.mark.parametrize("T,H,d,R,dv", [(32, 4, 40, 128, 48), (65, 8, 64, 256, 64), (300, 8, 64, 256, 64), (300, 16, 64, 256, 128)])
def test_heads_of_a_latent(T, H, d, R, dv):
    rng = np.random.default_rng(T + H)
    q, cache, gate = rng.standard_normal((T, H * d)).astype(np.float32), rng.standard_normal((T, R)).astype(np.float32), rng.standard_normal((T, H * dv)).astype(np.float32)
    uk, uv = bf16(rng.standard_normal((H * d, R)) / d ** 0.5), bf16(rng.standard_normal((H * dv, R)) / R ** 0.5)
    got = capi.latent_attend(q, cache, 0, H, d, 0, dv, R, uk, uv, R ** -0.5, gate=gate, w_bf16=True).reshape(T, H, dv)
    c = cache.astype(np.float64)
    for h in range(H):
        s = q[:, h * d:(h + 1) * d].astype(np.float64) @ uk[h * d:(h + 1) * d].astype(np.float64) @ c.T * R ** -0.5
        s[np.triu_indices(T, 1)] = -np.inf
        p = np.exp(s - s.max(axis=1, keepdims=True))
        want = p / p.sum(axis=1, keepdims=True) @ c @ uv[h * dv:(h + 1) * dv].T / (1 + np.exp(-gate[:, h * dv:(h + 1) * dv].astype(np.float64)))
        # a score of order one is off by the first product's bound, which moves the weights by as much; then the second's
        assert np.abs(got[:, h] - want).max() < 4 * (bound(d) + bound(R))
