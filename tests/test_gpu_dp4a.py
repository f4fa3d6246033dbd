"""The dp4a matvec (xalm_b200/csrc/matvec_idp.cuh) over unit-interleaved rows and the prompt's dequantiser of such rows: what the "mma" knob's 0 and 2 select, and what
rows too long or shards too narrow for the tensor-core matvec take."""
import numpy as np
import pytest

from oracle import oracle
from xalm_b200 import capi, types as T

from gpu_util import LOGIT_TOL, bits, greedy_compare, random_raw, synth_pair

pytestmark = pytest.mark.gpu

INT = [T.Q8_0, T.Q4_0, T.Q4_1, T.Q5_0, T.Q5_1, T.Q8]
PROMPT = [1, 84, 61, 35, 90, 107, 100, 119]


@pytest.fixture(autouse=True)
def dp4a():
    capi.tune("mma", 0)
    yield
    capi.tune("mma", 1)


@pytest.mark.parametrize("t", INT, ids=lambda t: t.name)
@pytest.mark.parametrize("d,n", [(64, 256), (32, 512), (128, 1024), (2432, 2048)])
def test_effective_weights_bit_exact(t, d, n):
    raw = random_raw(t, d, n, seed=11)
    W = oracle.dequant(t.id, raw, d * n).reshape(d, n)
    for j in (0, 15, 16, 31, 32, n // 2 + 5, n - 1):
        e = np.zeros(n, np.float32)
        e[j] = 1.0
        assert np.array_equal(capi.matmul(e, raw, t.id, n, d), W[:, j]), f"column {j}"


# a unit a row, part of a stage of 16 units, a stage, more than one; fewer rows than tiles for every SM, and more
@pytest.mark.parametrize("t", INT, ids=lambda t: t.name)
@pytest.mark.parametrize("d,n", [(32, 256), (96, 768), (4096, 4096), (1184, 4352), (2400, 14336), (32, 45056)])
def test_random_x_vs_oracle(t, d, n):
    raw = random_raw(t, d, n, seed=3)
    x = np.random.default_rng(4).standard_normal(n).astype(np.float32)
    y = capi.matmul(x, raw, t.id, n, d)
    ref = oracle.matmul(x, raw, t.id, n, d, acc_mode=2)
    scale = np.sqrt(n) * np.abs(oracle.dequant(t.id, raw[: t.nbytes(n)], n)).max()
    assert np.max(np.abs(y - ref)) <= 2e-6 * scale + 1e-6          # the bound of test_gpu_formats.py
    assert np.array_equal(bits(y), bits(capi.matmul(x, raw, t.id, n, d)))
    if n > 256:                                                    # sums in another order than the tensor-core matvec's: it is not that one
        capi.tune("mma", 1)
        longest = n > 44672                                        # that takes no such row: the same kernel whatever the knob says
        assert np.array_equal(bits(y), bits(capi.matmul(x, raw, t.id, n, d))) == longest


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("wtype", ["q8_0", "q8", "q4_0", "q5_1"])
def test_model_and_prompt(wtype, mode):
    """Tokens of single steps, and a batched prompt over unit rows (mode 2: the 4- and 5-bit formats stay fragment tiles)."""
    capi.tune("mma", mode)
    config, om, gm = synth_pair("tiny", wtype, seed=2, std=0.06)
    otoks, gtoks, maxdiff, margin = greedy_compare(config, om, gm, PROMPT, 16)
    assert maxdiff <= LOGIT_TOL and otoks == gtoks, f"min margin {margin}"
    toks = np.random.default_rng(1).integers(3, config["vocab_size"], 50).tolist()
    want = [om.forward(t, p, 1) for p, t in enumerate(toks)]
    assert np.max(np.abs(gm.prefill(toks, 0, 2) - np.stack(want))) <= LOGIT_TOL
    gm.close(); om.close()
