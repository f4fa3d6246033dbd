"""Whole models over passes long enough for the kernels of long passes: recurrences and delta rules by chunks of 64 tokens (rec_chunk.cu, delta_chunk.cu) with layers
of different shapes in one workspace, on the main stream and beside another branch; attention over a latent wider than 128 channels.  300 tokens go in
passes of 128, 128 and 44 (the last one token by token in the recurrences), then single tokens: the state is handed on in every way there is."""
import importlib

import numpy as np
import pytest

from xalm_b200 import capi
from xalm_b200.model import Model

pytestmark = pytest.mark.gpu

F32_TOL, BF16_TOL = 2e-4, 6e-2  # as in the families' own tests
N, STEPS, CHUNK = 300, 3, 128


def configs():
    K, D, B, P, A = (importlib.import_module(f"{f}_oracle") for f in ("kubolorn", "duletar", "bolovik", "pavitar", "nabalix"))
    n = dict(window=100, softcap=9.0)
    return {
        "kubolorn": (K, K.make_config(59, 64, [
            K.parallel_layer(4, 2, 32, 0.2, {"dims": 8, "base": 100.0}, 4, 32, 72, 2, 3, 2, 1.1, 0.7, mlp={"kind": "dense", "ff": 96}),
            K.gla_layer(2, 48, 64, 8.0, rank=8, mlp={"kind": "dense", "ff": 64}),
            K.gla_layer(3, 20, 12, 4.0, rank=4)], groups=2)),
        "duletar": (D, D.make_config(59, 64, [
            D.retention_layer(3, 16, 24, [0.9, 0.99, 0.5], rot_dims=8, base=200.0, mlp=D.dense(96)),
            D.gated_latent_layer(4, 16, 16, 136, 24, mlp=D.dense(64)),
            D.retention_layer(2, 80, 40, [1.0, 0.75]),
            D.latent_layer(3, 16, 8, 16, 192, 32, mlp=D.dense(64))])),
        "bolovik": (B, B.make_config(vocab=59, width=64, groups=2, layers=[
            B.delta_layer(4, 2, 16, 32, mlp=B.dense(96)),
            B.attention_layer(4, 2, 32, 32, window=90, keep_first=5, mlp=B.dense(64)),
            B.delta_layer(2, 2, 80, 24, conv=4)])),
        "pavitar": (P, P.make_config(59, 64, [
            P.latent_layer(4, 16, 16, 24, 136, 90, 0.25),
            P.attention_layer(4, 2, 32, 32, 100, 0.2, (100.0, 8)),
            P.latent_layer(6, 12, 20, 16, 320, 1000, 0.3)])),
        "nabalix": (A, A.make_config(vocab=59, width=64, streams=2, layers=[
            dict(n, H=4, G=2, d=32, dv=32, Hr=3, dr=16, dvr=24, ff=96),
            dict(n, H=2, G=1, d=16, dv=16, Hr=2, dr=96, dvr=64, ff=None)])),
    }


@pytest.fixture(scope="module", params=["kubolorn", "duletar", "bolovik", "pavitar", "nabalix"])
def case(request):
    O, cfg = configs()[request.param]
    W = O.random_weights(cfg, 5)
    tokens = np.random.default_rng(8).integers(0, cfg["vocab"], N + STEPS).tolist()
    logits = O.forward(cfg, W, tokens, {}) if request.param in ("kubolorn", "pavitar") else O.forward(cfg, W, tokens)
    return request.param, cfg, W, tokens, logits[0] if isinstance(logits, tuple) else logits


def run(cfg, W, tokens, precision, overlap=1):
    for k, v in (("seq_chunk", CHUNK), ("seq_overlap", overlap)):
        capi.tune(k, v)
    try:
        m = Model.from_json(cfg, W, "F32" if precision == capi.PRECISION_F32 else "BF16").cuda(max_tokens=N + STEPS, precision=precision)
        out = []
        for _ in range(2):  # again after a release: the workspace still holds what the first run left
            rows = [m.prefill(tokens[:N], 0, 2).reshape(N, -1)]
            rows += [m.prefill(tokens[p:p + 1], p, 1).reshape(1, -1) for p in range(N, N + STEPS)]
            out.append(np.concatenate(rows))
            m.release()
        m.close()
    finally:
        capi.tune("seq_chunk", 256)
        capi.tune("seq_overlap", 1)
    assert np.array_equal(out[0], out[1])
    return out[0]


@pytest.mark.parametrize("precision,tol", [(capi.PRECISION_F32, F32_TOL), (capi.PRECISION_BF16, BF16_TOL)])
def test_against_float64_and_without_branches(case, precision, tol):
    name, cfg, W, tokens, logits = case
    got = run(cfg, W, tokens, precision)
    assert got.shape == logits.shape
    assert np.abs(got - logits).max() / max(1.0, np.abs(logits).max()) < tol
    assert np.array_equal(got, run(cfg, W, tokens, precision, overlap=0))
