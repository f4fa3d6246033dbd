"""GEMMs of passes whose tiles are whole waves and a rest: the rest in clusters, a launch of its own where that pays, with ragged rows and columns, one tile behind the
wave and nearly a wave, and K too short for it."""
import numpy as np
import pytest

from xalm_b200 import capi, synth
from xalm_b200 import types as T

pytestmark = pytest.mark.gpu


def _fp16(x):
    return x.astype(np.float16).astype(np.float32)


@pytest.mark.parametrize("shape", [(2600, 4096, 2048), (1000, 2112, 5024), (385, 4096, 10016), (129, 4096, 19200), (140, 4096, 30016), (129, 576, 20000)])
@pytest.mark.parametrize("split", [1, 2, 3])
def test_rest_of_the_last_wave(shape, split):
    """Tolerance of the other GEMM tests (test_gpu_prefill.py): a share's sum is fp32 as the whole sum is, and there are at most 8 of them."""
    Tn, K, N = shape
    t = T.parse("f32")
    a, w = synth.normal(6, 81, Tn * K, 1.0).reshape(Tn, K), synth.normal(6, 82, N * K, 0.05).reshape(N, K)
    raw = np.ascontiguousarray(w).view(np.uint8).reshape(-1)
    out = capi.gemm(a, raw, t.id, K, N, split)
    rows = np.unique(np.r_[0:Tn:37, Tn - 1, 127, 128])  # (every column, rows of every tile)
    if split == 3:
        ref = a[rows].astype(np.float64) @ w.astype(np.float64).T
    else:
        hi = _fp16(a[rows])
        ref = (hi.astype(np.float64) + (_fp16(a[rows] - hi) if split == 2 else 0.0)) @ _fp16(w).astype(np.float64).T
    assert np.max(np.abs(out[rows] - ref)) <= 2e-5 * float(np.abs(ref).max()) + 1e-6
    assert np.array_equal(out, capi.gemm(a, raw, t.id, K, N, split))
