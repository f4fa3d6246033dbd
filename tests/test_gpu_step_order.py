"""One-token steps of config.json families: kernels that start while the one before still runs, branches on a second stream, steps replayed from a graph
with or without their copies.  None of it may change a bit of a result: the kernels and the order of their sums are the same."""
import importlib

import numpy as np
import pytest

from xalm_b200 import capi
from xalm_b200.model import InferenceState, Model

pytestmark = pytest.mark.gpu

FAMILIES = [("nabalix", "mixed3"), ("nabalix", "k64_tiles"), ("bolovik", "mixed"), ("bolovik", "k64_tiles"), ("duletar", "mixed"), ("duletar", "k64_tiles"),
            ("kubolorn", "mixed"), ("kubolorn", "k64_tiles"), ("mizerax", "mixed"), ("mizerax", "k64_tiles"), ("pavitar", "mixed"), ("pavitar", "k64_tiles")]
CHUNK = 16


def load(family, name, stream=None, **knobs):
    test = importlib.import_module(f"test_gpu_{family}")
    cfg = test.CONFIGS[name]
    for k, v in dict(knobs, seq_chunk=CHUNK).items():
        capi.tune(k, v)
    return cfg["vocab"], Model.from_json(cfg, test.O.random_weights(cfg, 3), "BF16").cuda(max_tokens=160, stream=stream)


@pytest.fixture(autouse=True)
def knobs_as_they_were():
    yield
    for k, v in dict(pdl=1, seq_graph=1, seq_overlap=1, seq_chunk=256).items():
        capi.tune(k, v)


def run(m, vocab):
    """Logits of a prompt's last position, of single steps, of every position of a pass and one token more, and that call's probabilities."""
    rng = np.random.default_rng(5)
    toks = rng.integers(0, vocab, 160).tolist()
    state, out = InferenceState(m.config), []
    out.append(m.prefill(toks[:40], 0, 1))
    p = 40
    for _ in range(6):
        m.forward(state, toks[p], p)
        out.append(state.logits().copy())
        p += 1
    out.append(m.prefill(toks[p:p + CHUNK + 1], p, 2).reshape(-1))
    p += CHUNK + 1
    lg, pr = m.prefill(toks[p:p + CHUNK + 1], p, 2, targets=toks[p + 1:p + CHUNK + 2])
    out += [lg.reshape(-1), pr]
    e = np.exp(lg.astype(np.float64) - lg.max(1, keepdims=True))
    want = e[np.arange(CHUNK + 1), toks[p + 1:p + CHUNK + 2]] / e.sum(1)
    assert np.abs(pr / want - 1).max() < 1e-5  # exponentials in fp32 of differences below 2^5
    m.release()
    out.append(m.prefill(toks[:1], 0, 1))  # a sequence that starts with a single token
    return np.concatenate([np.ravel(a) for a in out])


@pytest.mark.parametrize("family,name", FAMILIES)
def test_dependents_graphs_and_branches_do_not_change_a_bit(family, name):
    got = {}
    for pdl in (1, 0):
        for graph in (1, 0):
            for overlap in (1, 0):
                vocab, m = load(family, name, pdl=pdl, seq_graph=graph, seq_overlap=overlap)
                got[pdl, graph, overlap] = run(m, vocab)
                m.close()
    for k, v in got.items():
        assert np.array_equal(v, got[1, 1, 1]), f"pdl, seq_graph, seq_overlap = {k} changed the results"


@pytest.mark.parametrize("family,name", FAMILIES)
def test_steps_that_are_waited_for_between_steps_that_are_not_on_a_callers_stream(family, name):
    import torch

    vocab, m = load(family, name)
    toks = np.random.default_rng(6).integers(0, vocab, 60).astype(np.int32)
    state, want = InferenceState(m.config), []
    for p in range(60):
        m.forward(state, int(toks[p]), p)
        want.append(state.logits().copy())
    m.close()
    stream = torch.cuda.Stream()
    vocab, m = load(family, name, stream=stream.cuda_stream)
    state, p = InferenceState(m.config), 0
    while p < 60:
        for _ in range(min(p % 4, 59 - p)):  # these lie in the stream when the next step is enqueued
            m.forward_async(int(toks[p]), p)
            p += 1
        if p % 3:
            m.forward(state, int(toks[p]), p)
            lg = state.logits()
        else:
            lg = m.prefill(toks[p:p + 1], p, 1)
        assert np.array_equal(lg, want[p])
        p += 1
        if p < 57:
            m.prefill_async(toks[p:p + 1], p, 0)
            p += 1
    m.close()
