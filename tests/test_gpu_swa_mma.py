"""Attention of passes of many tokens on the tensor cores (queries and probabilities as three bf16 planes): heads whose channels do not fill a tile, passes and
keys around the tiles, every mask and term of the score, and its error beside that of fp32 sums."""
import numpy as np
import pytest

from test_gpu_swa_one import bf16, inputs, reference
from xalm_b200 import capi

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
