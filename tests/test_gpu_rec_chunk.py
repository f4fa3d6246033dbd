"""Gated linear recurrences of long passes (rec_chunk.cu) against float64, and against the token-by-token kernels on the same inputs cut short.

Tolerance: a value is a sum of at most T d products whose terms have signs, formed in fp32; its distance from float64 stays within a few times that of the
token-by-token kernels, measured here on the same inputs (the two differ in the order of the sums only)."""
import numpy as np
import pytest

from xalm_b200 import capi

pytestmark = pytest.mark.gpu

CUT = 79  # the longest pass that goes token by token
MODES = ["gla", "ssd", "hgrn2", "retention"]


def softplus(x):
    return np.logaddexp(0.0, x)


def case(mode, T, H, d, dv, seed=0, small=False):
    """(arguments by name, per-token arrays among them, decays f, writes g, queries q as float64 (T, H, d))."""
    rng = np.random.default_rng([seed, T, d, dv])
    n = lambda *s: rng.standard_normal(s).astype(np.float32)
    q, k, v = n(T, H * d), n(T, H * d), n(T, H * dv)
    q64, k64 = (x.astype(np.float64).reshape(T, H, d) for x in (q, k))
    if mode == "gla":
        f = 1.0 / (1.0 + np.exp(-(n(T, H * d) * (4.0 if small else 1.0) + (0.0 if small else 3.0))))
        f = f.astype(np.float32)
        return dict(q=q, k=k, v=v, f=f), f.astype(np.float64).reshape(T, H, d), k64, q64 * d ** -0.5
    if mode == "ssd":
        f, bias, A = n(T, H), 0.2 * n(H), n(H) - (0.0 if small else 1.5)
        dt = softplus(f.astype(np.float64) + bias)
        dec = np.exp(-np.exp(A.astype(np.float64)) * dt)[:, :, None] * np.ones((1, 1, d))
        return dict(q=q, k=k, v=v, f=f, dt_bias=bias, A_log=A, skip=n(H)), dec, dt[:, :, None] * k64, q64
    if mode == "hgrn2":
        bias, low = n(H * d), np.float32(0.0 if small else 0.5) * rng.random(H * d).astype(np.float32)
        f = low + (1.0 - low) / (1.0 + np.exp(-(k.astype(np.float64) + bias)))
        f = f.reshape(T, H, d)
        return dict(qz=q, fz=k, v=v, f_bias=bias, lower=low), f, 1.0 - f, q64 / (1.0 + np.exp(-q64))
    dec = (rng.random(H) * 0.1 + (0.0 if small else 0.9)).astype(np.float32)
    return dict(q=q, k=k, v=v, decay=dec), np.ones((T, H, d)) * dec.astype(np.float64)[None, :, None], k64 * d ** -0.5, q64


def call(mode, a, lo, hi, state, H, d, dv, norm=None, gate=None):
    cut = {k: (x[lo:hi] if k in ("q", "k", "v", "f", "qz", "fz") else x) for k, x in a.items()}
    if mode == "hgrn2":
        return capi.hgrn2(cut["qz"], cut["fz"], cut["v"], state, H, d, dv, f_bias=a["f_bias"], lower=a["lower"], norm_w=norm)
    if mode == "retention":
        return capi.retention(cut["q"], cut["k"], cut["v"], state, H, d, dv, a["decay"], gate=None if gate is None else gate[lo:hi], eps=1e-5)
    return capi.keyed_recurrence(cut["q"], cut["k"], cut["v"], cut["f"], state, H, 1, d, dv, 1 if mode == "gla" else 2, q_scale=d ** -0.5 if mode == "gla" else 0.0,
                                 dt_bias=a.get("dt_bias"), A_log=a.get("A_log"), skip=a.get("skip"), norm_w=norm, gate=None if gate is None else gate[lo:hi])


def by_tokens(mode, a, T, state, H, d, dv, **kw):
    out, st = [], state
    for lo in range(0, T, CUT):
        o, st = call(mode, a, lo, min(T, lo + CUT), st, H, d, dv, **kw)
        out.append(o)
    return np.concatenate(out), st


def exact(mode, a, f, g, q, state, norm=None, gate=None):
    T, H, d = f.shape
    v = a["v"].astype(np.float64).reshape(T, H, -1)
    S, out = state.astype(np.float64), []
    for t in range(T):
        S = f[t][:, :, None] * S + g[t][:, :, None] * v[t][:, None, :]
        o = np.einsum("hij,hi->hj", S, q[t])
        if "skip" in a:
            o = o + a["skip"].astype(np.float64)[:, None] * v[t]
        if norm is not None or mode == "retention":
            o = o / np.sqrt((o * o).mean(-1, keepdims=True) + 1e-5) * (1.0 if norm is None else norm)
        if gate is not None:
            z = gate[t].astype(np.float64).reshape(H, -1)
            o = o * z / (1.0 + np.exp(-z))
        out.append(o.reshape(-1))
    return np.stack(out), S


def off(x, ref):
    return np.linalg.norm(np.asarray(x, np.float64) - ref) / np.linalg.norm(ref)


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("T,H,d,dv", [(80, 2, 64, 128), (128, 3, 64, 64), (97, 2, 16, 20), (129, 1, 128, 128), (200, 2, 68, 100), (577, 2, 64, 128)])
@pytest.mark.parametrize("small", [False, True])  # decays near zero: products of 64 of them underflow
def test_chunks(mode, T, H, d, dv, small):
    a, f, g, q = case(mode, T, H, d, dv, small=small)
    rng = np.random.default_rng(5)
    s0 = rng.standard_normal((H, d, dv)).astype(np.float32)
    kw = {}
    if mode != "ssd":
        kw["norm"] = (1.0 + 0.1 * rng.standard_normal(dv)).astype(np.float32) if mode != "retention" else None
        kw["gate"] = rng.standard_normal((T, H * dv)).astype(np.float32) if mode in ("gla", "retention") else None
    want, s_want = exact(mode, a, f, g, q, s0, **kw)
    got, s_got = call(mode, a, 0, T, s0, H, d, dv, **kw)
    tok, s_tok = by_tokens(mode, a, T, s0, H, d, dv, **kw)
    assert off(got, want) <= 2.0 * off(tok, want) + 2e-7, (off(got, want), off(tok, want))
    assert off(s_got, s_want) <= 2.0 * off(s_tok, s_want) + 2e-7, (off(s_got, s_want), off(s_tok, s_want))
    again, s_again = call(mode, a, 0, T, s0, H, d, dv, **kw)
    assert np.array_equal(got, again) and np.array_equal(s_got, s_again)


@pytest.mark.parametrize("mode", ["gla", "ssd"])
def test_infinities_stay_with_the_tokens_that_see_them(mode):
    T, H, d, dv = 150, 2, 64, 128
    a, f, g, q = case(mode, T, H, d, dv)
    clean = call(mode, a, 0, T, np.zeros((H, d, dv)), H, d, dv)[0]
    for name, at in (("v", 70), ("k", 100), ("q", 37)):
        b = dict(a)
        b[name] = a[name].copy()
        b[name][at, 5] = np.inf
        got = call(mode, b, 0, T, np.zeros((H, d, dv)), H, d, dv)[0]
        assert np.array_equal(got[:at], clean[:at]), name
        assert not np.isfinite(got[at]).all(), name
        if name == "q":
            assert np.array_equal(got[at + 1:], clean[at + 1:])
