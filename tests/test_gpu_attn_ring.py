"""Steps of models whose attention runs as clusters (four and eight query heads per kv head), in and past their window: what such a kernel fetches ahead of its wait is
all but the row that this step writes and the sinks that it rotates again; those are fetched behind it."""
import numpy as np
import pytest

from xalm_b200 import capi
from xalm_b200.model import InferenceState

from gpu_util import LOGIT_TOL, greedy_compare, synth_pair

pytestmark = pytest.mark.gpu


# windows below, at and above a unit of 16 slots, and of several: every kv_pos of a round is met
@pytest.mark.parametrize("context,steps", [(6, 30), (16, 40), (17, 40), (50, 120)])
@pytest.mark.parametrize("hd,nh,nkv", [(32, 8, 2), (64, 8, 2), (128, 8, 2), (32, 8, 1), (64, 16, 2), (128, 8, 1), (256, 8, 1)])
def test_past_the_window(hd, nh, nkv, context, steps):
    config, om, gm = synth_pair("tiny", "f16", seed=5, std=(nh * hd) ** -0.5, context=context, dim=nh * hd, hidden_dim=2 * nh * hd, n_heads=nh, n_kv_heads=nkv, head_dim=hd, n_layers=2)
    otoks, gtoks, maxdiff, margin = greedy_compare(config, om, gm, [1, 266, 267], steps)
    assert maxdiff <= LOGIT_TOL and otoks == gtoks, f"min margin {margin}"
    for layer in range(config["n_layers"]):
        for which in (0, 1):
            a, b = (m(layer, which).view(np.float16).astype(np.float32) for m in (gm.read_kv, om.kv))
            assert np.max(np.abs(a - b)) <= 2e-3 * max(1.0, np.abs(b).max())
            # Rounded to fp16 once, so that only values within fp32 rounding of a boundary differ: but for the sinks, which are rotated and rounded again at every step, and
            # for the layers behind their attention
            assert layer or np.mean((a != b).reshape(context, -1)[2:]) < 0.02
    gm.close(); om.close()


def test_more_slots_than_a_cluster_holds_at_once():
    """1030 and more slots: every warp of a cluster of 16 refills its ring, and the ring of the cache turns over."""
    config, om, gm = synth_pair("tiny", "f16", seed=6, std=1024 ** -0.5, context=1100, dim=1024, hidden_dim=2048, n_heads=8, n_kv_heads=2, head_dim=128, n_layers=1, max_seq_len=1100)
    prompt = np.random.default_rng(3).integers(3, config["vocab_size"], 1085).tolist()
    otoks, gtoks, maxdiff, margin = greedy_compare(config, om, gm, prompt, 40)
    assert maxdiff <= LOGIT_TOL and otoks == gtoks, f"min margin {margin}"
    gm.close(); om.close()


@pytest.mark.parametrize("nh,nkv", [(8, 2), (8, 1)])
def test_steps_in_flight(nh, nkv):
    """Enqueued without a wait in between, each step's early fetches overlap the step before: the same bits as one by one, past the window too."""
    config, om, gm = synth_pair("tiny", "f16", seed=7, std=1024 ** -0.5, context=40, dim=1024, hidden_dim=2048, n_heads=nh, n_kv_heads=nkv, head_dim=128, n_layers=4)
    toks = np.random.default_rng(2).integers(3, config["vocab_size"], 120).tolist()
    state, kv = InferenceState(config), []
    for waits in (True, False):
        for pos, t in enumerate(toks):
            if waits:
                gm.forward(state, t, pos, 1)
            else:
                gm.forward_async(t, pos, 1)
        gm.sync()
        kv.append([gm.read_kv(layer, which).copy() for layer in range(4) for which in (0, 1)] + [gm.read_state(capi.S_LOGITS, config["vocab_size"])])
    assert all(np.array_equal(a, b) for a, b in zip(*kv))
    gm.close(); om.close()


@pytest.mark.parametrize("nh,nkv", [(8, 2), (8, 1)])
def test_graph_and_programmatic_launches_change_no_bit(nh, nkv):
    outs = []
    try:
        for graph, pdl in ((1, 1), (0, 1), (1, 0), (0, 0)):
            capi.tune("graph", graph)
            capi.tune("pdl", pdl)
            config, om, gm = synth_pair("tiny", "q8_0", seed=6, std=0.06, context=20, n_heads=nh, n_kv_heads=nkv, head_dim=32, n_layers=3)
            state, seq = InferenceState(config), []
            for pos, tok in enumerate([1, 84, 61, 35, 90, 107, 100, 119, 7, 9, 300, 2] * 3):
                gm.forward(state, tok, pos, 1)
                seq.append(state.logits().copy())
            outs.append(np.stack(seq))
            gm.close(); om.close()
    finally:
        capi.tune("graph", 1)
        capi.tune("pdl", 1)
    assert all(np.array_equal(outs[0], o) for o in outs[1:])
