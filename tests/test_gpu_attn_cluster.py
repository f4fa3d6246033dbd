"""One-token attention as a cluster of CTAs per kv head (xalm_b200/csrc/attn_cluster.cu) against float64 and, for what is not finite, against the split kernel."""
import numpy as np
import pytest

from xalm_b200 import capi
from xalm_b200.model import InferenceState

from gpu_util import synth_pair

pytestmark = pytest.mark.gpu


def both(q, k, v, hd, n, nh, nkv):
    out = []
    for on in (0, 1):
        capi.tune("attn_cluster", on)
        out.append(capi.mha(q, k.view(np.uint16), v.view(np.uint16), hd, n, len(k), nh, nkv))
    capi.tune("attn_cluster", 1)
    return out


def inputs(hd, n, nh, nkv, seed, scale=1.0):
    r = np.random.default_rng(seed)
    return ((scale * r.standard_normal(nh * hd)).astype(np.float32), *(r.standard_normal((n + 3, nkv * hd)).astype(np.float16) for _ in range(2)))


# one slot; the ends of a 16-slot unit; one unit for every warp of a cluster of 16 (1024 slots) and one more; long enough for the ring to be refilled
@pytest.mark.parametrize("n", [1, 15, 16, 17, 257, 1024, 1025, 3001])
@pytest.mark.parametrize("hd,nh,nkv", [(128, 32, 8), (128, 8, 1), (64, 8, 2), (32, 8, 1), (256, 16, 2), (128, 80, 20)])
def test_against_float64(hd, nh, nkv, n):
    q, k, v = inputs(hd, n, nh, nkv, n + hd, scale=2.0)
    got = both(q, k, v, hd, n, nh, nkv)[1]
    K, V = (a[:n].astype(np.float64).reshape(n, nkv, hd) for a in (k, v))
    for h in range(nh):
        s = K[:, h // (nh // nkv)] @ q[h * hd:(h + 1) * hd].astype(np.float64) / np.sqrt(hd)
        p = np.exp(s - s.max())
        want = p / p.sum() @ V[:, h // (nh // nkv)]
        # fp32: a score of up to 10 is off by some of its last bits (2^-24 each), which moves its weight by as much; sums of weights times values of order 1
        assert np.max(np.abs(got[h * hd:(h + 1) * hd] - want)) < 64 * 10 * 2.0 ** -24


@pytest.mark.parametrize("what", ["key inf", "key -inf", "key nan", "value inf", "value -inf", "value nan", "query inf", "query nan", "query large", "query tiny"])
def test_what_is_not_finite_goes_where_the_split_kernel_sends_it(what):
    hd, n, nh, nkv = 128, 300, 32, 8
    q, k, v = inputs(hd, n, nh, nkv, 5)
    kind, val = what.split()
    if kind == "query":
        if val in ("inf", "nan"):
            q[5] = float(val)
        else:
            q *= 1e30 if val == "large" else 1e-30
    else:
        (k if kind == "key" else v)[77, 3 * hd + 9] = float(val)
    a, b = both(q, k, v, hd, n, nh, nkv)
    for f in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(f(a), f(b))
    fin = np.isfinite(a)
    assert np.max(np.abs(a[fin] - b[fin])) < 64 * 10 * 2.0 ** -24


# the first slot of all, of a warp's unit (16, 64), inside a unit, the last; alone, and as the only key of its warp (n = 17)
@pytest.mark.parametrize("hd,nh,nkv", [(128, 32, 8), (64, 32, 4)])
@pytest.mark.parametrize("n,slot", [(1, 0), (17, 0), (17, 16), (300, 0), (300, 16), (300, 64), (300, 77), (300, 299)])
@pytest.mark.parametrize("what", ["key nan", "key inf", "key -inf", "value nan", "value inf"])
def test_what_is_not_finite_at_any_slot(what, n, slot, hd, nh, nkv):
    """Against IEEE arithmetic in float64: a score that is NaN or +inf makes its head NaN, one that is -inf weighs nothing, a value reaches its own channel."""
    q, k, v = inputs(hd, n, nh, nkv, 11)
    kind, val = what.split()
    (k if kind == "key" else v)[slot, 3 * hd + 9] = float(val)
    got = both(q, k, v, hd, n, nh, nkv)[1].reshape(nh, hd)
    K, V = (a[:n].astype(np.float64).reshape(n, nkv, hd) for a in (k, v))
    with np.errstate(invalid="ignore"):
        for h in range(nh):
            s = K[:, h // (nh // nkv)] @ q[h * hd:(h + 1) * hd].astype(np.float64) / np.sqrt(hd)
            p = np.exp(s - s.max())
            want = p / p.sum() @ V[:, h // (nh // nkv)]
            for f in (np.isnan, np.isposinf, np.isneginf):
                assert np.array_equal(f(got[h]), f(want))
            fin = np.isfinite(want)
            assert not fin.any() or np.max(np.abs(got[h][fin] - want[fin])) < 64 * 10 * 2.0 ** -24  # as above


@pytest.mark.parametrize("hd,nh,nkv", [(128, 160, 40), (64, 320, 80), (32, 304, 38), (256, 640, 80)])
def test_many_kv_heads_are_the_split_kernels(hd, nh, nkv):
    """Fewer than four CTAs per kv head: slower than the split kernel on short contexts.  The kernels add in another order, so equal bits are the same kernel."""
    assert np.array_equal(*both(*inputs(hd, 100, nh, nkv, 2), hd, 100, nh, nkv))
    assert not np.array_equal(*both(*inputs(hd, 100, nh // nkv * 8, 8, 2), hd, 100, nh // nkv * 8, 8))


@pytest.mark.parametrize("graph", [1, 0])
@pytest.mark.parametrize("cluster", [1, 0])
def test_the_timeline_has_every_layers_attention(cluster, graph):
    """Of steps that were captured before it began to record as of others; and no step afterwards is another one."""
    capi.tune("attn_cluster", cluster)
    config, om, gm = synth_pair("small", "q8_0", seed=1, std=0.03)   # four query heads per kv head
    capi.tune("attn_cluster", 1)
    capi.tune("graph", graph)
    try:
        state, logits = InferenceState(config), []
        for again in range(2):
            gm.forward(state, 5, 0, 1)
            capi.timeline_start(400)
            for call in (lambda: gm.forward(state, 6, 1, 1), lambda: (gm.forward_async(6, 1, 1), gm.sync())):
                call()
                logits.append(gm.read_state(capi.S_LOGITS, config["vocab_size"]))
            rec = capi.timeline_stop(400)
            at = rec[rec[:, 0] == 300].astype(np.int64)
            assert len(at) == 2 * config["n_layers"]
            assert np.all(at[:, 1] <= at[:, 2]) and np.all(at[:, 2] <= at[:, 3]) and np.all(at[1:, 1] > at[:-1, 1])
        gm.forward(state, 6, 1, 1)
        logits.append(state.logits().copy())
        assert all(np.array_equal(a, logits[0]) for a in logits)
    finally:
        capi.tune("graph", 1)
        capi.timeline_start(0)
    gm.close(); om.close()
