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
