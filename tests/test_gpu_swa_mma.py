"""Attention of passes of many tokens on the tensor cores (queries and probabilities as three bf16 planes): heads whose channels do not fill a tile, passes and
keys around the tiles, every mask and term of the score, and its error beside that of fp32 sums."""
import numpy as np
import pytest

import bolovik_oracle as O
from test_gpu_swa_one import bf16, inputs, reference
from xalm_b200 import capi
from xalm_b200.model import Model

pytestmark = pytest.mark.gpu

# exact products, fp32 sums over d <= 128 channels and up to a few hundred keys in blocks: a few dozen roundings of 2^-24 of values of order one, and
# exponentials of differences below 2^5 (as in the one-token kernel)
TOL = 2e-5


@pytest.mark.parametrize("H,G,d,dv", [(1, 1, 32, 32), (4, 2, 64, 64), (3, 1, 72, 40), (2, 2, 128, 128), (10, 2, 40, 128), (2, 1, 128, 64), (160, 2, 32, 32)])
@pytest.mark.parametrize("T,pos0", [(16, 0), (17, 3), (64, 0), (65, 63), (31, 130)])
def test_shapes(H, G, d, dv, T, pos0):
    q, k, v = inputs(T, pos0 + T, H, G, d, dv, H * d + T)
    got = capi.swa_attention(q * np.float32(1.001), k, v, pos0, H, G, d, dv, 10 ** 6, d ** -0.5, cache_bf16=True)
    assert np.abs(got - reference(q * np.float32(1.001), k, v, pos0, H, G, 10 ** 6, scale=d ** -0.5)).max() < TOL


@pytest.mark.parametrize("pos0", [0, 70, 300])
@pytest.mark.parametrize("T", [16, 100])
def test_every_mask_and_term_of_the_score(pos0, T):
    H, G, d, rng = 4, 2, 32, np.random.default_rng(pos0 + T)
    q, k, v = inputs(T, pos0 + T, H, G, d, d, pos0)
    u = [rng.uniform(0.1, 1, H).astype(np.float32) for _ in range(4)]
    gate, heads = rng.standard_normal((T, H * d)).astype(np.float32), rng.standard_normal((T, H)).astype(np.float32)
    got = capi.swa_attention(q, k, v, pos0, H, G, d, d, 90, 0.2, softcap=5.0, r1=u[0], r2=u[1], gate=gate, cache_bf16=True)
    assert np.abs(got - reference(q, k, v, pos0, H, G, 90, scale=0.2, softcap=5.0, r=u, gate=gate)).max() < TOL
    got = capi.biased_attention(q, k, v, pos0, H, G, d, d, 0.2, slope=u[2], sink=u[3], gate=heads, cache_bf16=True)
    assert np.abs(got - reference(q, k, v, pos0, H, G, 10 ** 6, scale=0.2, slope=u[2], sink=u[3], gate=heads)).max() < TOL
    got = capi.swa_attention_kept(q, k, v, pos0, H, G, d, d, 50, 9, 0.2, cache_bf16=True)
    assert np.abs(got - reference(q, k, v, pos0, H, G, 50, keep=9, scale=0.2)).max() < TOL
    for chunk in (1, 64, 130):
        got = capi.chunked_attention(q, k, v, pos0, H, G, d, d, chunk, 0.2, cache_bf16=True)
        assert np.abs(got - reference(q, k, v, pos0, H, G, 10 ** 6, chunk=chunk, scale=0.2)).max() < TOL


def test_no_further_from_float64_than_fp32_sums():
    """The same bf16 keys and values in an fp32 cache take the fp32 FMA kernel."""
    H, G, d, T, pos0 = 4, 1, 128, 128, 1400
    q, k, v = inputs(T, pos0 + T, H, G, d, d, 7)
    q = q * np.float32(1.001)
    want = reference(q, k, v, pos0, H, G, 10 ** 6, scale=d ** -0.5)
    err = [np.linalg.norm(capi.swa_attention(q, k, v, pos0, H, G, d, d, 10 ** 6, d ** -0.5, cache_bf16=c) - want) / np.linalg.norm(want) for c in (True, False)]
    assert err[0] <= err[1]


@pytest.mark.parametrize("T,pos0", [(16, 0), (16, 1040), (32, 330), (45, 63), (64, 512), (100, 29), (130, 700)])
@pytest.mark.parametrize("n_splits", [2, 5, 16])
def test_keys_split_over_several_ctas(T, pos0, n_splits):
    """Splits of whole key blocks: fewer blocks than splits, one block each, several each; every term that is applied where the splits are joined."""
    H, G, d, dv, rng = 4, 2, 40, 64, np.random.default_rng(T + pos0)
    q, k, v = inputs(T, pos0 + T, H, G, d, dv, T + pos0)
    sink, slope = rng.uniform(0.1, 1, H).astype(np.float32), rng.uniform(0.01, 0.1, H).astype(np.float32)
    wide, heads = rng.standard_normal((T, H * dv)).astype(np.float32), rng.standard_normal((T, H)).astype(np.float32)
    kw = dict(n_splits=n_splits, cache_bf16=True)
    for window in (10 ** 6, 90):
        want = reference(q, k, v, pos0, H, G, window, scale=0.2, softcap=5.0, gate=wide)
        assert np.abs(capi.swa_attention(q, k, v, pos0, H, G, d, dv, window, 0.2, softcap=5.0, gate=wide, **kw) - want).max() < TOL
    want = reference(q, k, v, pos0, H, G, 10 ** 6, scale=0.2, slope=slope, sink=sink, gate=heads)
    assert np.abs(capi.biased_attention(q, k, v, pos0, H, G, d, dv, 0.2, slope=slope, sink=sink, gate=heads, **kw) - want).max() < TOL
    want = reference(q, k, v, pos0, H, G, 50, keep=9, scale=0.2)
    assert np.abs(capi.swa_attention_kept(q, k, v, pos0, H, G, d, dv, 50, 9, 0.2, **kw) - want).max() < TOL
    want = reference(q, k, v, pos0, H, G, 10 ** 6, chunk=64, scale=0.2)
    assert np.abs(capi.chunked_attention(q, k, v, pos0, H, G, d, dv, 64, 0.2, **kw) - want).max() < TOL


@pytest.mark.parametrize("T", [16, 33, 64])
@pytest.mark.parametrize("n_splits", [1, 4])
def test_a_ring_that_has_wrapped(T, n_splits):
    """The window's keys lie around the ring's end, behind slots of first positions that stay."""
    H, G, d, pos0, window = 2, 1, 64, 1000, 150
    q, k, v = inputs(T, pos0 + T, H, G, d, d, T)
    for ring in (window - 1 + T, 257):
        got = capi.swa_attention(q, k, v, pos0, H, G, d, d, window, 0.2, ring=ring, n_splits=n_splits, cache_bf16=True)
        assert np.abs(got - reference(q, k, v, pos0, H, G, window, scale=0.2)).max() < TOL
        got = capi.swa_attention_kept(q, k, v, pos0, H, G, d, d, window, 7, 0.2, ring=ring, n_splits=n_splits, cache_bf16=True)
        assert np.abs(got - reference(q, k, v, pos0, H, G, window, keep=7, scale=0.2)).max() < TOL


def test_splits_are_split():
    """The sums of three splits, joined, are not those of one walk over the keys."""
    q, k, v = inputs(40, 640, 4, 2, 64, 64, 5)
    got = [capi.swa_attention(q, k, v, 600, 4, 2, 64, 64, 10 ** 6, 0.125, n_splits=s, cache_bf16=True) for s in (1, 3)]
    assert not np.array_equal(*got) and np.abs(got[0] - got[1]).max() < TOL


@pytest.mark.parametrize("limit,joins", [(64, 0), (100, 0), (128, 1), (4096, 1)])
def test_a_short_pass_over_a_long_cache_splits_the_keys(limit, joins):
    """8 CTAs of queries and heads, and a cache of `limit` slots: from two key blocks on the pass has a join's kernel."""
    cfg = O.make_config(vocab=50, width=64, layers=[O.attention_layer(8, 2, 32, 32, mlp=O.dense(64))], groups=2)
    count = []
    for n in (64, limit):
        m = Model.from_json(cfg, O.random_weights(cfg, 1), "BF16").cuda(max_tokens=n)
        m.prefill(np.arange(20), 0, want_logits=0)
        count.append(m.last_launch_count())
        m.close()
    assert count[1] == count[0] + joins


@pytest.mark.parametrize("T,pos0,n_splits", [(64, 0, 1), (64, 0, 2), (100, 30, 1), (20, 200, 3)])
@pytest.mark.parametrize("what", ["v inf", "v nan", "k inf", "q inf"])
def test_infinities_and_nan_stay_with_the_queries_that_see_them(T, pos0, n_splits, what):
    """A masked key's weight is zero, and zero times its value must not count; an infinite key whose score is minus infinity has no weight either."""
    H, G, d = 2, 1, 64
    q, k, v = inputs(T, pos0 + T, H, G, d, d, T)
    j = pos0 + T // 2  # a position inside the pass
    if what == "q inf":
        q[T // 2, 3] = np.inf
    else:
        (v if what[0] == "v" else k)[[j, j - pos0 // 2], 3] = np.nan if what == "v nan" else np.inf
    with np.errstate(invalid="ignore"):
        for kw in (dict(), dict(window=20), dict(chunk=16)):
            window, chunk = kw.get("window", 10 ** 6), kw.get("chunk", 0)
            want = reference(q, k, v, pos0, H, G, window, chunk=chunk, scale=0.125)
            if chunk:
                got = capi.chunked_attention(q, k, v, pos0, H, G, d, d, chunk, 0.125, n_splits=n_splits, cache_bf16=True)
            else:
                got = capi.swa_attention(q, k, v, pos0, H, G, d, d, window, 0.125, n_splits=n_splits, cache_bf16=True)
            assert np.isfinite(want).any() and not np.isfinite(want).all()
            assert np.allclose(got, want, rtol=0, atol=TOL, equal_nan=True)


@pytest.mark.parametrize("T", [5, 9, 15])
@pytest.mark.parametrize("H,G,d,dv", [(3, 1, 40, 40), (4, 2, 72, 40), (2, 2, 128, 128), (1, 1, 32, 32)])
def test_passes_of_a_few_tokens(H, G, d, dv, T):
    """Tiles of mostly padding, warps without a query; short caches in one piece and long ones whose keys are split."""
    for pos0, splits in ((0, 1), (3, 2), (700, 5), (1500, 7)):
        q, k, v = inputs(T, pos0 + T, H, G, d, dv, H * d + T)
        want = reference(q * np.float32(1.001), k, v, pos0, H, G, 10 ** 6, scale=d ** -0.5)
        got = capi.swa_attention(q * np.float32(1.001), k, v, pos0, H, G, d, dv, 10 ** 6, d ** -0.5, n_splits=splits, cache_bf16=True)
        assert np.abs(got - want).max() < TOL
        got = capi.swa_attention_kept(q, k, v, pos0, H, G, d, dv, 50, 9, 0.2, n_splits=splits, cache_bf16=True)
        assert np.abs(got - reference(q, k, v, pos0, H, G, 50, keep=9, scale=0.2)).max() < TOL


@pytest.mark.parametrize("T,pos0,n_splits", [(5, 0, 1), (9, 300, 4), (15, 70, 1)])
@pytest.mark.parametrize("what", ["v inf", "v nan", "k inf", "q inf"])
def test_infinities_and_nan_in_passes_of_a_few_tokens(T, pos0, n_splits, what):
    test_infinities_and_nan_stay_with_the_queries_that_see_them(T, pos0, n_splits, what)
