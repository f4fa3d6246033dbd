"""Calls of the Llama family that wait for their token (xalm_cuda_forward): its parameters and logits go through pinned memory, and a call without a buffer for
the logits leaves them on the device."""
import numpy as np
import pytest

from xalm_b200 import capi
from xalm_b200.model import InferenceState

from gpu_util import synth_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [512, 1056])   # a part of a CTA of the kernel that takes them out, and one CTA and a rest
def test_logits_reach_the_host_only_when_asked_for(vocab):
    config, om, gm = synth_pair("tiny", "q8_0", seed=4, std=0.06, vocab_size=vocab)
    L = capi.lib()
    pinned = np.ctypeslib.as_array(L.xalm_cuda_logits_host(gm._h), shape=(vocab,))
    state = InferenceState(config)
    om.forward(7, 0, 1)
    gm.forward(state, 7, 0, 1)
    kept = state.logits().copy()
    assert np.array_equal(pinned, kept)
    want = om.forward(9, 1, 1)
    capi.check(L.xalm_cuda_forward(gm._h, 9, 1, 1, None))
    assert np.array_equal(pinned, kept)                                     # as it was
    on_device = gm.read_state(capi.S_LOGITS, vocab)
    assert np.max(np.abs(on_device - want)) < 1e-2 and not np.array_equal(on_device, kept)
    om.forward(11, 2, 0)
    gm.forward(state, 11, 2, 0)                                             # no classifier: nothing moves
    assert np.array_equal(pinned, kept)
    want = om.forward(13, 3, 1)
    gm.forward(state, 13, 3, 1)
    assert np.array_equal(state.logits(), pinned) and np.max(np.abs(pinned - want)) < 1e-2
    gm.close(); om.close()
