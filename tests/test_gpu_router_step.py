"""Router of a one-token step (moe_router_step_kernel: up to 32 experts whose rows fit shared memory) and of longer passes: row lengths around a round of 2048 channels,
one expert to more than 32, every score and choice against a restatement in float64."""
import numpy as np
import pytest

from xalm_b200 import capi

pytestmark = pytest.mark.gpu


def bf16(a):
    return (np.ascontiguousarray(a, np.float32).view(np.uint32) + 0x8000 & 0xFFFF0000).view(np.float32)


@pytest.mark.parametrize("K", [8, 64, 1024, 2048, 2056, 4096])
@pytest.mark.parametrize("E,top", [(1, 1), (4, 2), (10, 3), (16, 4), (20, 20), (32, 4), (33, 4)])
@pytest.mark.parametrize("T", [1, 5, 40])
def test_choice_and_weights(E, top, K, T):
    rng = np.random.default_rng(E * K + T)
    h, wr = rng.standard_normal((T, K)).astype(np.float32), bf16(3 * rng.standard_normal((E, K)) / K ** 0.5)
    ff = 8
    wg, wu, wd = (bf16(rng.standard_normal(s)) for s in ((E, ff, K), (E, ff, K), (E, K, ff)))
    idx, wgt, _ = capi.moe_ffn(h, wr, wg, wu, wd, top, w_bf16=True)
    z = h.astype(np.float64) @ wr.T.astype(np.float64)
    s = 1 / (1 + np.exp(-z))
    order = np.argsort(-s, axis=1, kind="stable")[:, :top]
    gap = np.diff(np.sort(s, axis=1), axis=1).min(axis=1) if E > 1 else np.ones(T)
    clear = gap > 1e-5   # scores that fp32 sums cannot mistake for one another
    assert clear.any()
    assert np.array_equal(idx[clear], order[clear])
    assert np.abs(wgt - np.take_along_axis(s, idx, 1)).max() < 1e-5


@pytest.mark.parametrize("score,group,renorm", [("softmax", "max", True), ("softmax", "top2", False), ("sigmoid", "top2", True), ("sigmoid", "max", False)])
@pytest.mark.parametrize("E,top,n_groups,keep", [(16, 4, 4, 2), (8, 2, 4, 2), (12, 3, 1, 1), (30, 5, 3, 1), (32, 8, 8, 3)])
def test_groups_and_scores(E, top, n_groups, keep, score, group, renorm):
    K, ff = 256, 8
    rng = np.random.default_rng(E + top)
    for _ in range(8):
        h, wr = rng.standard_normal((1, K)).astype(np.float32), bf16(3 * rng.standard_normal((E, K)) / K ** 0.5)
        wg, wu, wd = (bf16(rng.standard_normal(s)) for s in ((E, ff, K), (E, ff, K), (E, K, ff)))
        idx, wgt, _, _ = capi.moe_ffn_routed(h, wr, wg, wu, wd, top, n_groups=n_groups, keep_groups=keep, score=score, group=group, renormalise=renorm, w_bf16=True)
        z = (h.astype(np.float64) @ wr.T.astype(np.float64))[0]
        s = np.exp(z - z.max()) / np.exp(z - z.max()).sum() if score == "softmax" else 1 / (1 + np.exp(-z))
        if n_groups > 1:
            parts = np.sort(s.reshape(n_groups, -1), axis=1)
            best = np.argsort(-(parts[:, -1] if group == "max" or parts.shape[1] == 1 else parts[:, -1] + parts[:, -2]), kind="stable")[:keep]
            allowed = np.isin(np.arange(E) // (E // n_groups), best)
        else:
            allowed = np.ones(E, bool)
        want = np.argsort(np.where(allowed, -s, np.inf), kind="stable")[:top]
        assert np.array_equal(idx[0], want)   # (random scores: no two within fp32 rounding)
        w = s[want] / s[want].sum() if renorm else s[want]
        assert np.abs(wgt[0] - w).max() < 1e-5


# What is not finite, against the kernel of longer passes (two equal tokens): NaN rows (which have no place in an order: that kernel's choice is the rule), infinite
# scores of either sign and infinities in the token, whose sigmoids are ties
@pytest.mark.parametrize("E,top", [(4, 2), (16, 4), (31, 5), (32, 32)])
@pytest.mark.parametrize("what", ["nan row 0", "nan row 3", "nan row last", "nan rows", "all nan", "inf row", "inf token", "huge token"])
@pytest.mark.parametrize("score,groups", [("sigmoid", 0), ("softmax", 0), ("softmax", 4)])
def test_what_is_not_finite_as_in_longer_passes(E, top, what, score, groups):
    if groups and E % groups:
        pytest.skip("experts do not form that many groups")
    K, ff = 128, 8
    rng = np.random.default_rng(E)
    h, wr = rng.standard_normal((1, K)).astype(np.float32), bf16(3 * rng.standard_normal((E, K)) / K ** 0.5)
    if what == "all nan":
        h[0, 3] = np.nan
    elif what == "nan rows":
        wr[1::3, 5] = np.nan
    elif what.startswith("nan row"):
        wr[{"0": 0, "3": 3, "last": E - 1}[what.split()[-1]], 7] = np.nan
    elif what == "inf row":
        wr[2, 7], wr[1, 7] = np.inf, -np.inf
    elif what == "inf token":
        h[0, 9] = np.inf
    else:
        h *= 1e30
    wg, wu, wd = (bf16(rng.standard_normal(s)) for s in ((E, ff, K), (E, ff, K), (E, K, ff)))
    # (two groups of two experts hold too few for the largest choices)
    kw = dict(n_groups=groups, keep_groups=max(2, -(-top * groups // E)) if groups else 0, score=score, group="max", renormalise=True, w_bf16=True)
    one = capi.moe_ffn_routed(h, wr, wg, wu, wd, top, **kw)
    two = capi.moe_ffn_routed(np.repeat(h, 2, axis=0), wr, wg, wu, wd, top, **kw)
    assert np.array_equal(one[0][0], two[0][0]) and np.array_equal(np.isnan(one[1][0]), np.isnan(two[1][0]))
    fin = np.isfinite(two[1][0])
    assert np.abs(one[1][0][fin] - two[1][0][fin]).max(initial=0) < 1e-5


@pytest.mark.parametrize("E,top,K", [(32, 4, 2480), (32, 32, 64), (1, 1, 40000), (8, 3, 8192)])   # the first two: as many rows, and as many bytes, as it takes
@pytest.mark.parametrize("bad", [None, "nan", "inf"])
def test_plain_logits_with_bias_and_gate(E, top, K, bad):
    rng = np.random.default_rng(K + E)
    h, wr, gate = rng.standard_normal((1, K)).astype(np.float32), bf16(3 * rng.standard_normal((E, K)) / K ** 0.5), bf16(rng.standard_normal(K) / K ** 0.5)
    bias = rng.standard_normal(E).astype(np.float32)
    if bad:
        bias[E // 2] = float(bad)
    ff = 8
    wg, wu, wd = (bf16(rng.standard_normal(s) / K ** 0.5) for s in ((E, ff, K), (E, ff, K), (E, K, ff)))
    x, base = np.zeros((1, K), np.float32), np.ones((1, K), np.float32)
    one = capi.moe_chosen(x, h, wr, wg, wu, wd, top, bias=bias, base=base, gate_row=gate, w_bf16=True)
    r2 = lambda a: np.repeat(a, 2, axis=0)
    two = capi.moe_chosen(r2(x), r2(h), wr, wg, wu, wd, top, bias=bias, base=r2(base), gate_row=gate, w_bf16=True)
    assert np.array_equal(one[1][0], two[1][0]) and np.array_equal(np.isnan(one[2][0]), np.isnan(two[2][0]))
    if bad:
        return
    z = (h.astype(np.float64) @ wr.T.astype(np.float64))[0] + bias
    want = np.argsort(-z, kind="stable")[:top]
    w = np.exp(z[want] - z[want[0]])
    assert np.array_equal(one[1][0], want) and np.abs(one[2][0] - w / w.sum()).max() < 1e-5
    assert np.abs(one[0] - two[0][:1]).max() < 1e-4   # sums of up to 32 rows of order one, and the gate's
