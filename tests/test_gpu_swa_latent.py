"""Attention of passes of several tokens over a latent (one head whose first channels are the values) on the tensor cores, against float64 and the fp32 kernels."""
import numpy as np
import pytest

import duletar_oracle as O
from xalm_b200 import capi

pytestmark = pytest.mark.gpu

# exact products, fp32 sums over up to 576 channels and 800 keys in blocks, values of order one
TOL = 4e-5


def inputs(T, n, H, d, dv, R, r=0, seed=0):
    rng = np.random.default_rng([seed, T, n, R])
    q = rng.standard_normal((T, H * (d + r)))
    c = O.bf16_round(rng.standard_normal((n, R + r)))
    uk, uv = rng.standard_normal((H * d, R)) * R ** -0.5, rng.standard_normal((H * dv, R)) * R ** -0.5
    return tuple(np.asarray(x, np.float32) for x in (q, c, uk, uv))


def reference(q, c, uk, uv, pos0, H, d, dv, R, scale, window, gate=None, freqs=None):
    T, n, r = q.shape[0], c.shape[0], c.shape[1] - R
    q, c, uk, uv = (np.asarray(x, np.float64) for x in (q, c, uk, uv))
    q = q.reshape(T, H, d + r)
    qr = O.rotate(q[:, :, d:], np.arange(pos0, pos0 + T), freqs) if r else q[:, :, d:]
    i, j = np.arange(pos0, pos0 + T)[:, None], np.arange(n)[None]
    seen = (j <= i) & (i - j < window)
    out = np.zeros((T, H, dv))
    for h in range(H):
        s = q[:, h, :d] @ (c[:, :R] @ uk[h * d:(h + 1) * d].T).T + qr[:, h] @ c[:, R:].T
        s = np.where(seen, s * scale, -np.inf)
        p = np.exp(s - s.max(1, keepdims=True))
        p /= p.sum(1, keepdims=True)
        v = c[:, :R] @ uv[h * dv:(h + 1) * dv].T
        out[:, h] = np.stack([p[t][seen[t]] @ v[seen[t]] for t in range(T)])
        if gate is not None:
            out[:, h] /= 1.0 + np.exp(-np.asarray(gate, np.float64)[:, h, None])
    return out.reshape(T, H * dv)


@pytest.mark.parametrize("H,R", [(1, 136), (3, 256), (16, 200), (8, 320), (5, 512), (16, 384)])
@pytest.mark.parametrize("T,pos0,splits", [(5, 0, 0), (9, 700, 0), (33, 62, 3), (64, 130, 0), (100, 300, 1)])
def test_window(H, R, T, pos0, splits):
    d = dv = 16
    q, c, uk, uv = inputs(T, pos0 + T, H, d, dv, R)
    gate = np.random.default_rng(1).standard_normal((T, H)).astype(np.float32)
    for window, g, ring in ((10 ** 6, None, None), (70, gate, 69 + T)):
        got = capi.latent_window(q, c, pos0, H, d, dv, R, uk, uv, 0.3, window, g, ring, splits, cache_bf16=True)
        assert np.abs(got - reference(q, c, uk, uv, pos0, H, d, dv, R, 0.3, window, g)).max() < TOL


@pytest.mark.parametrize("H,R,r", [(4, 256, 64), (2, 512, 64), (3, 136, 8), (2, 250, 6)])  # the last one's rows are no whole 16-byte pieces: the general kernels
@pytest.mark.parametrize("T,pos0", [(6, 90), (40, 0), (65, 300)])
def test_rotated_part(H, R, r, T, pos0):
    d = dv = 24
    q, c, uk, uv = inputs(T, pos0 + T, H, d, dv, R, r)
    freqs = O.rotary_frequencies(r, 10000.0)
    cc = np.array(c)
    got = capi.latent_attend(q, cc, pos0, H, d, r, dv, R, uk, uv, 0.2, freqs, cache_bf16=True)
    assert np.abs(got - reference(q, c, uk, uv, pos0, H, d, dv, R, 0.2, 10 ** 6, freqs=freqs)).max() < TOL


def test_no_further_from_float64_than_fp32_sums():
    """The same bf16 rows in an fp32 cache take the fp32 FMA kernel."""
    H, d, R, T, pos0 = 4, 64, 512, 64, 700
    q, c, uk, uv = inputs(T, pos0 + T, H, d, d, R)
    want = reference(q, c, uk, uv, pos0, H, d, d, R, d ** -0.5, 10 ** 6)
    err = [np.linalg.norm(capi.latent_window(q, c, pos0, H, d, d, R, uk, uv, d ** -0.5, 10 ** 6, cache_bf16=b) - want) / np.linalg.norm(want) for b in (True, False)]
    assert err[0] <= 1.05 * err[1], err


@pytest.mark.parametrize("T,pos0,splits", [(40, 0, 1), (100, 30, 2), (9, 200, 3)])
@pytest.mark.parametrize("what", ["c inf", "c nan", "q inf"])
def test_infinities_and_nan_stay_with_the_queries_that_see_them(T, pos0, splits, what):
    H, d, R = 4, 32, 256
    q, c, uk, uv = inputs(T, pos0 + T, H, d, d, R)
    j = pos0 + T // 2
    if what == "q inf":
        q[T // 2, 3] = np.inf
    else:
        c[j, 3] = np.inf if what == "c inf" else np.nan
    for window in (10 ** 6, 20):
        with np.errstate(invalid="ignore"):
            want = reference(q, c, uk, uv, pos0, H, d, d, R, 0.2, window)
        got = capi.latent_window(q, c, pos0, H, d, d, R, uk, uv, 0.2, window, n_splits=splits, cache_bf16=True)
        fine = np.isfinite(want)
        assert fine.any() and not fine.all()
        assert np.abs(got[fine] - want[fine]).max() < TOL and not np.isfinite(got[~fine]).any()
