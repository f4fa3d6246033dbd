"""Attention of one-to-four-token steps (clusters of CTAs per key/value group) at its edges: heads per group around the heads of a CTA, channel counts
around a chunk of lanes, key counts around the CTAs, units and blocks of a cluster, both cache types, every term of the score."""
import numpy as np
import pytest

from xalm_b200 import capi

pytestmark = pytest.mark.gpu


def reference(q, k, v, pos0, H, G, window, chunk=0, keep=0, scale=1.0, softcap=0.0, r=None, slope=None, sink=None, gate=None):
    T, n = q.shape[0], k.shape[0]
    q, k, v = (a.astype(np.float64) for a in (q.reshape(T, H, -1), k.reshape(n, G, -1), v.reshape(n, G, -1)))
    out = np.zeros((T, H, v.shape[2]))
    for t in range(T):
        i, j = pos0 + t, np.arange(pos0 + t + 1)
        seen = j[((i - j < window) | (j < keep)) & ((j // chunk == i // chunk) if chunk else True)]
        for h in range(H):
            s = k[seen, h * G // H] @ q[t, h] * scale
            if softcap:
                s = softcap * np.tanh(s / softcap)
            if r is not None:
                s = s - r[0][h] * np.log1p(r[1][h] * (i - seen))
            if slope is not None:
                s = s - slope[h] * (i - seen)
            m = s.max() if sink is None else max(s.max(), sink[h])
            e = np.exp(s - m)
            out[t, h] = e @ v[seen, h * G // H] / (e.sum() + (0 if sink is None else np.exp(sink[h] - m)))
    out = out.reshape(T, -1)
    return out if gate is None else out / (1 + np.exp(-np.repeat(gate, out.shape[1] // gate.shape[1], 1)))


def bf16(a):
    return (np.ascontiguousarray(a, np.float32).view(np.uint32) + 0x8000 & 0xFFFF0000).view(np.float32)


# values of order one, softmax weights summing to one: the products' fp32 sums over d <= 768 channels and the weights' exponentials of differences
# below 2^5 leave 2^-24 * (sqrt(768) * 4 + 2^5) = 9e-6
TOL = 2e-5


def inputs(T, n, H, G, d, dv, seed):
    rng = np.random.default_rng(seed)
    return [bf16(rng.standard_normal(s)) for s in ((T, H * d), (n, G * d), (n, G * dv))]


@pytest.mark.parametrize("H,G,d,dv", [(1, 1, 8, 8), (2, 1, 64, 64), (6, 2, 72, 40), (10, 2, 128, 128), (3, 3, 136, 8), (8, 2, 256, 256), (4, 2, 64, 264), (2, 2, 520, 768),
                                      (5, 1, 768, 512), (12, 4, 24, 136)])
@pytest.mark.parametrize("T,pos0,splits", [(1, 0, 1), (1, 6, 1), (2, 7, 2), (1, 511, 1), (4, 130, 3)])
def test_shapes(H, G, d, dv, T, pos0, splits):
    q, k, v = inputs(T, pos0 + T, H, G, d, dv, H * d + pos0)
    for cache in (False, True):
        got = capi.swa_attention(q, k, v, pos0, H, G, d, dv, 10 ** 6, d ** -0.5, n_splits=splits, cache_bf16=cache)
        assert np.abs(got - reference(q, k, v, pos0, H, G, 10 ** 6, scale=d ** -0.5)).max() < TOL


@pytest.mark.parametrize("pos0", [3, 64, 1500])
@pytest.mark.parametrize("splits", [1, 3])
def test_every_term_of_the_score(pos0, splits):
    H, G, d, T, rng = 6, 2, 32, 2, np.random.default_rng(pos0)
    q, k, v = inputs(T, pos0 + T, H, G, d, d, pos0)
    u = [rng.uniform(0.1, 1, H).astype(np.float32) for _ in range(4)]
    gate, heads = rng.standard_normal((T, H * d)).astype(np.float32), rng.standard_normal((T, H)).astype(np.float32)
    got = capi.swa_attention(q, k, v, pos0, H, G, d, d, 700, 0.2, softcap=5.0, r1=u[0], r2=u[1], gate=gate, n_splits=splits)
    assert np.abs(got - reference(q, k, v, pos0, H, G, 700, scale=0.2, softcap=5.0, r=u, gate=gate)).max() < TOL
    got = capi.biased_attention(q, k, v, pos0, H, G, d, d, 0.2, slope=u[2], sink=u[3], gate=heads, n_splits=splits)
    assert np.abs(got - reference(q, k, v, pos0, H, G, 10 ** 6, scale=0.2, slope=u[2], sink=u[3], gate=heads)).max() < TOL
    got = capi.swa_attention_kept(q, k, v, pos0, H, G, d, d, 50, 9, 0.2, n_splits=splits)
    assert np.abs(got - reference(q, k, v, pos0, H, G, 50, keep=9, scale=0.2)).max() < TOL
    got = capi.chunked_attention(q, k, v, pos0, H, G, d, d, 130, 0.2, n_splits=splits)
    assert np.abs(got - reference(q, k, v, pos0, H, G, 10 ** 6, chunk=130, scale=0.2)).max() < TOL


@pytest.mark.parametrize("H,R", [(1, 136), (16, 256), (3, 512), (8, 640)])
@pytest.mark.parametrize("pos0", [0, 9, 700])
def test_latent_rows_serve_as_keys_and_values(H, R, pos0):
    rng, d, T = np.random.default_rng(R + pos0), 8, 1
    q, cache = bf16(rng.standard_normal((T, H * d))), bf16(rng.standard_normal((pos0 + T, R)))
    uk, uv = bf16(rng.standard_normal((H * d, R)) / R ** 0.5), bf16(rng.standard_normal((H * d, R)) / R ** 0.5)
    k, v = cache.astype(np.float64) @ uk.T, cache.astype(np.float64) @ uv.T
    for bf in (False, True):
        got = capi.latent_window(q, cache, pos0, H, d, d, R, uk, uv, d ** -0.5, 300, cache_bf16=bf)
        assert np.abs(got - reference(q, k, v, pos0, H, H, 300, scale=d ** -0.5)).max() < 2 * TOL  # two more products of R channels
