"""The tensor-core matvec (xalm_b200/csrc/matvec_mma.cuh) on rows that fill a ring stage (64 block columns of the 8-bit formats, 128 of the others), a part
of one, or end inside the 64 records that are unrolled."""
import numpy as np
import pytest

from oracle import oracle
from xalm_b200 import capi, types as T

from gpu_util import random_raw

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1024, 2016, 2048, 2080, 3072, 4064, 4096, 6176])   # 32, 63, 64, 65, 96, 127, 128, 193 block columns
@pytest.mark.parametrize("t", [T.Q8_0, T.Q4_0, T.Q4_1, T.Q5_0, T.Q5_1, T.Q8], ids=lambda t: t.name)
def test_rows_that_end_inside_a_stage(t, n):
    d = 32
    raw = random_raw(t, d, n, seed=n)
    x = np.random.default_rng(n + 1).standard_normal(n).astype(np.float32)
    ref = oracle.matmul(x, raw, t.id, n, d, acc_mode=2)
    scale = np.sqrt(n) * np.abs(oracle.dequant(t.id, raw[: t.nbytes(n)], n)).max()
    # x enters with 23 bits of its block's largest value and the sums are fp32: the bound of test_gpu_formats.py
    assert np.max(np.abs(capi.matmul(x, raw, t.id, n, d) - ref)) <= 2e-6 * scale + 1e-6


# the longest rows that stages of half the records leave room for, and a hidden size whose rows are not whole 256-element units: the fallback is the kernel of the
# planar layout there, whose sums differ in their last bits
@pytest.mark.parametrize("t,n", [(T.Q4_0, 37184), (T.Q4_1, 36384), (T.Q5_0, 35552), (T.Q5_1, 34752), (T.Q5_1, 29568), (T.Q4_0, 28672), (T.Q5_0, 24608), (T.Q8_0, 28704), (T.Q8, 36000)],
                         ids=lambda a: getattr(a, "name", a))
def test_longest_rows(t, n):
    d = 32
    raw = random_raw(t, d, n, seed=n)
    x = np.random.default_rng(n).standard_normal(n).astype(np.float32)
    ref = oracle.matmul(x, raw, t.id, n, d, acc_mode=2)
    scale = np.sqrt(n) * np.abs(oracle.dequant(t.id, raw[: t.nbytes(n)], n)).max()
    got = {}
    for mode in (0, 1):
        capi.tune("mma", mode)
        got[mode] = capi.matmul(x, raw, t.id, n, d)
    assert np.max(np.abs(got[1] - ref)) <= 2e-6 * scale + 1e-6  # as above
    assert not np.array_equal(got[0], got[1]), "not the tensor-core matvec"
