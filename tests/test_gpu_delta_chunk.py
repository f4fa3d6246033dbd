"""The gated delta rule of long passes (delta_chunk.cu) against float64, and against the token-by-token kernel on the same inputs cut short.

Tolerance: both form fp32 sums of the same products in another order, so that the chunked kernels' distance from float64 stays within a small multiple of the
token-by-token kernel's, measured here on the same inputs."""
import numpy as np
import pytest

import bolovik_oracle as O
from xalm_b200 import capi

pytestmark = pytest.mark.gpu

CUT = 63  # the longest pass that goes token by token


def case(T, H, G, d, dv, taps, like=False, seed=0):
    rng = np.random.default_rng([seed, T, d, dv])
    n = lambda *s: rng.standard_normal(s).astype(np.float32)
    nq, nv = G * d, H * dv
    x = dict(q=n(T, nq), k=n(T, nq), v=n(T, nv), gate=n(T, nv), b=2 * n(T, H), a=2 * n(T, H))
    if like:  # keys that hardly differ: every token rewrites what the one before it wrote
        x["k"] = (2.0 + 0.1 * n(T, nq)).astype(np.float32)
    par = dict(wq=0.6 * n(nq, taps), wk=(np.abs(n(nq, taps)) if like else 0.6 * n(nq, taps)), wv=0.6 * n(nv, taps), A_log=n(H) - (5 if like else 1), dt_bias=n(H), norm_w=1 + 0.2 * n(dv), eps=1e-5)
    return x, par, 0.3 * n(H, d, dv), n(taps - 1, 2 * nq + nv)


def run(x, par, s, c, lo, hi, H, G, d, dv):
    return capi.delta_rule(*(x[k][lo:hi] for k in ("q", "k", "v", "gate", "b", "a")), s, c, H, G, d, dv, **par)


def off(x, ref):
    return np.linalg.norm(np.asarray(x, np.float64) - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("T,H,G,d,dv,taps", [(64, 2, 1, 64, 128, 4), (65, 3, 3, 16, 20, 3), (127, 2, 2, 128, 128, 1), (128, 12, 6, 64, 128, 4), (200, 2, 1, 100, 72, 5),
                                             (321, 12, 4, 128, 128, 4)])
@pytest.mark.parametrize("like", [False, True])
def test_chunks(T, H, G, d, dv, taps, like):
    x, par, s0, c0 = case(T, H, G, d, dv, taps, like)
    want, s_want, c_want = O.delta_rule(*(x[k] for k in ("q", "k", "v", "gate", "b", "a")), s0, c0, H=H, G=G, d=d, dv=dv, **par)
    got, s_got, c_got = run(x, par, s0, c0, 0, T, H, G, d, dv)
    outs, st, cs = [], s0, c0
    for lo in range(0, T, CUT):
        o, st, cs = run(x, par, st, cs, lo, min(T, lo + CUT), H, G, d, dv)
        outs.append(o)
    tok = np.concatenate(outs)
    assert off(got, want) <= 2.0 * off(tok, want) + 3e-7, (off(got, want), off(tok, want))
    assert off(s_got, s_want) <= 2.0 * off(st, s_want) + 3e-7, (off(s_got, s_want), off(st, s_want))
    if taps > 1:
        assert np.array_equal(c_got, cs)
    again = run(x, par, s0, c0, 0, T, H, G, d, dv)
    assert np.array_equal(got, again[0]) and np.array_equal(s_got, again[1])


def test_infinities_stay_with_the_tokens_that_see_them():
    T, H, G, d, dv, taps = 150, 2, 1, 64, 128, 4
    x, par, s0, c0 = case(T, H, G, d, dv, taps)
    clean = run(x, par, s0, c0, 0, T, H, G, d, dv)[0]
    for name, at in (("v", 70), ("k", 100), ("q", 37)):
        b = dict(x)
        b[name] = x[name].copy()
        b[name][at, 5] = np.inf
        got = run(b, par, s0, c0, 0, T, H, G, d, dv)[0]
        assert np.array_equal(got[:at], clean[:at]), name
        assert not np.isfinite(got[at:at + taps]).all(), name
        if name == "q":
            assert np.array_equal(got[at + taps:], clean[at + taps:])
