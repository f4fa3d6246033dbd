"""What the tensor-core GEMM does to a product on its way out, against the plain product followed by the elementwise kernel, and against float64.

The two paths form the same sums in the same order and apply the same functions, compiled in two kernels: their results differ by the contraction of a multiply
and an add at most, a few units in the last place of the function's largest term.  K = 64: one CTA per tile; K = 4096: a cluster shares a tile's K steps, and its
CTAs the columns."""
import numpy as np
import pytest

import duletar_oracle as O
from xalm_b200 import capi

pytestmark = pytest.mark.gpu

KINDS = [("add", 0), ("cap", 0), ("relu2", 0), ("gelu", 0), ("glu", 0), ("glu", 1), ("glu", 2)]
LIMIT = 1.5


def sigmoid(z):
    return 1.0 / (1.0 + np.exp(-z))


def gelu(z):
    return 0.5 * z * (1.0 + np.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))


def reference(kind, act, v, add):
    if kind == "add":
        return v + add
    if kind == "cap":
        return LIMIT * np.tanh(v / LIMIT)
    if kind == "relu2":
        return np.maximum(v, 0.0) ** 2
    if kind == "gelu":
        return gelu(v)
    g, u = v[:, 0::2], v[:, 1::2]
    if act == 0:
        g, u = np.minimum(g, LIMIT), np.clip(u, -LIMIT, LIMIT)
        return g * sigmoid(1.702 * g) * (u + 1.0)
    return (g * sigmoid(g) if act == 1 else gelu(g)) * u


def inputs(T, N, K):
    rng = np.random.default_rng([T, N, K])
    x = np.asarray(rng.standard_normal((T, K)), np.float16).astype(np.float32)  # exact in one plane
    w = O.bf16_round(1.4 * rng.standard_normal((N, K)) / np.sqrt(K))
    return x, np.asarray(w, np.float32), rng.standard_normal((T, N)).astype(np.float32)


@pytest.mark.parametrize("kind,act", KINDS)
@pytest.mark.parametrize("T", [1, 33, 130])
@pytest.mark.parametrize("N", [4, 260, 1028])
@pytest.mark.parametrize("K", [64, 4096])
def test_kinds(kind, act, T, N, K):
    N = N + 4 if kind == "glu" else N  # pairs of columns, four at a time
    x, w, add = inputs(T, N, K)
    want = reference(kind, act, x.astype(np.float64) @ np.asarray(w, np.float16).astype(np.float64).T, add)
    for planes in (1, 2):
        got, apart = (capi.rows_tc(x, w, kind, act, LIMIT, 1.702, add, planes, fused) for fused in (True, False))
        top = max(1.0, np.abs(want).max())
        assert np.abs(got - apart).max() <= 2.0 ** -21 * top
        # fp32 sums of K products of values of order one, in the tensor cores' truncating additions: 1e-6 a 16-product step, at random; slopes of the functions below 16
        assert np.abs(got - want).max() <= 16 * 2e-6 * np.sqrt(K / 16) * top


@pytest.mark.parametrize("kind,act", KINDS)
@pytest.mark.parametrize("K", [64, 4096])
def test_values_that_are_not_finite_stay_in_their_row(kind, act, K):
    x, w, add = inputs(40, 264, K)
    clean = capi.rows_tc(x, w, kind, act, LIMIT, 1.702, add, 1, True)
    x[7, 3], x[21, 5] = np.inf, np.nan
    got, apart = (capi.rows_tc(x, w, kind, act, LIMIT, 1.702, add, 1, fused) for fused in (True, False))
    rest = np.setdiff1d(np.arange(40), [7, 21])
    assert np.array_equal(got[rest], clean[rest])
    for row in (7, 21):
        assert np.array_equal(np.isnan(got[row]), np.isnan(apart[row])) and np.array_equal(np.isposinf(got[row]), np.isposinf(apart[row]))
