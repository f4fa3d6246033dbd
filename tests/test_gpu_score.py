"""Target probabilities of config.json families (prefill with targets): the device kernel against softmax in float64 over the same pass's logits."""
import ctypes as C

import numpy as np
import pytest

import bolovik_oracle as O
from xalm_b200 import capi
from xalm_b200.model import Model

pytestmark = pytest.mark.gpu


def small_model(vocab, chunk, max_tokens=96):
    cfg = O.make_config(vocab=vocab, width=64, layers=[O.attention_layer(4, 2, 16, 16, mlp=O.dense(64))], groups=2)
    capi.tune("seq_chunk", chunk)
    m = Model.from_json(cfg, O.random_weights(cfg, vocab)).cuda(max_tokens=max_tokens)
    capi.tune("seq_chunk", 256)
    return m


# below one value per thread, 16-byte rows with and without a remainder of the unrolled loop, rows that cannot be read 16 bytes at a time
@pytest.mark.parametrize("vocab", [3, 500, 2048, 8192 + 4 * 513, 10007])
@pytest.mark.parametrize("fetch", [False, True])
def test_target_probabilities_over_several_passes(vocab, fetch):
    rng = np.random.default_rng(vocab)
    m, n = small_model(vocab, 32), 75
    toks, targets = rng.integers(0, vocab, n), rng.integers(0, vocab, n)
    lg = m.prefill(toks, 0, want_logits=2).astype(np.float64)
    m.release()
    got_lg, got = m.prefill(toks, 0, want_logits=2, targets=targets, fetch_logits=fetch)
    assert got_lg is None or np.array_equal(got_lg, lg.astype(np.float32))
    e = np.exp(lg - lg.max(1, keepdims=True))
    want = e[np.arange(n), targets] / e.sum(1)
    # exp in fp32 on differences below 32: 2^-23 * 32 / 2 from rounding the difference, and as much from the sums of up to 10^4 terms in parts
    assert np.abs(got / want - 1).max() < 1e-5
    m.close()


def test_a_target_out_of_range_is_refused_after_the_rows_before_it():
    m, n = small_model(100, 32), 40
    toks = np.arange(n) % 100
    targets = toks.copy()
    targets[35] = 100
    with pytest.raises(capi.XalmError, match="target 100 out of range"):
        m.prefill(toks, 0, want_logits=2, targets=targets, fetch_logits=False)
    assert m.info("position") == n
    m.close()


@pytest.mark.parametrize("n,bad", [(75, 70), (75, 40), (40, 32), (110, 109)])
@pytest.mark.parametrize("what", ["token", "target"])
def test_a_failing_pass_leaves_the_probabilities_of_the_rows_before_it(n, bad, what):
    """Passes of 32.  A token that is out of range fails before its pass, a target after the rows before it."""
    rng = np.random.default_rng(n + bad)
    m = small_model(100, 32, 128)
    toks, targets = rng.integers(0, 100, n).astype(np.int32), rng.integers(0, 100, n).astype(np.int32)
    want = m.prefill(toks, 0, want_logits=2, targets=targets, fetch_logits=False)[1]
    m.release()
    (toks if what == "token" else targets)[bad] = 100
    got = np.full(n, -1, np.float32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    assert capi.lib().xalm_cuda_prefill(m._h, p(toks), n, 0, 2, None, p(targets), p(got)) != 0
    rows = bad // 32 * 32 if what == "token" else bad
    assert np.array_equal(got[:rows], want[:rows]) and (got[rows:] == -1).all()
    assert m.info("position") == (rows if what == "token" else min(n, bad // 32 * 32 + 32))
    m.close()


def test_the_limit_of_positions_costs_no_memory_where_the_caches_are_windowed():
    """A pass's probabilities need room for a pass.  Entries for every position up to the limit would be 1 GB on the device and 0.5 GB of pinned memory here."""
    import torch

    cfg = O.make_config(vocab=100, width=64, layers=[O.attention_layer(4, 2, 16, 16, window=32, mlp=O.dense(64))], groups=2)
    free = []
    for limit in (96, 96, 1 << 27):  # the first one loads the library's kernels
        m = Model.from_json(cfg, O.random_weights(cfg, 1)).cuda(max_tokens=limit)
        free.append(torch.cuda.mem_get_info()[0])
        toks = np.arange(80) % 100
        got = m.prefill(toks, 0, want_logits=2, targets=toks, fetch_logits=False)[1]
        assert ((got > 0) & (got < 1)).all()
        m.close()
    assert free[1] - free[2] < 64 << 20
