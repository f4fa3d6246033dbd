#!/usr/bin/env python
"""Golden vectors of the REFERENCE's own forward pass (jubruckne/Xalm src/infer.cpp, model.cpp, sampler.cpp), generated by
running the unmodified reference C++ — compiled by oracle/Makefile.ref behind the NEON / <print> shims — on small checkpoints.

Needs the reference's tree in /root/reference:

    make -f oracle/Makefile.ref && python tests/golden/make_ref_forward.py

Each case follows main.cpp:94-115: the prompt goes through Model::forward with HYDRATE_KV_CACHE (last prompt token with
OUTPUT_LOGITS), then greedy decoding with Sampler::sample_argmax.  Stored per case (tests/golden/ref_fwd_<case>.npz):
  tokens      prompt + greedy tokens chosen by the reference
  logits      (steps, vocab) fp32 — InferenceState::logits() after every OUTPUT_LOGITS forward
  probs       Sampler::sample_prob(token chosen, state) per step
  k_<l>/v_<l> fp16 bits of every layer's KV cache at the end (ring buffer + re-rotated sinks included)
  x           the residual stream after the last forward
and what is needed to rebuild the checkpoint on any box: a golden file name, or (shape, type, seed, std, overrides) for
xalm_b200.synth.write_checkpoint (deterministic).  tests/test_reference_forward.py checks the oracle restatement against
these on CPU and the CUDA path against them on the GPU.
"""
import ctypes as C
import json
import os
import sys
import tempfile

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(os.path.dirname(HERE))
sys.path.insert(0, ROOT)
from xalm_b200 import synth  # noqa: E402

CASES = [
    # name, source, context (-T), prompt, greedy steps
    dict(name="tiny_f16", file="tiny_f16.xalm", context=0, prompt=[1, 266, 267, 268, 269], steps=24),
    dict(name="tiny_bf16", file="tiny_bf16.xalm", context=0, prompt=[1, 266, 267, 268, 269], steps=24),
    dict(name="tiny_f8_e4m3", file="tiny_f8_e4m3.xalm", context=0, prompt=[1, 266, 267, 268, 269], steps=24),
    dict(name="tiny_f16_T6", file="tiny_f16.xalm", context=6, prompt=[1, 266, 267], steps=30),          # ring buffer + 2 sinks
    dict(name="synth_tiny_f32", synth=dict(shape="tiny", wtype="f32", seed=3, std=0.06), context=0, prompt=[1, 84, 61, 35, 90, 107, 100, 119], steps=16),
    dict(name="synth_tiny_f8_e5m2", synth=dict(shape="tiny", wtype="f8_e5m2", seed=4, std=0.06), context=0, prompt=[1, 84, 61, 35, 90, 107, 100, 119], steps=16),
    dict(name="synth_tiny_q8", synth=dict(shape="tiny", wtype="q8", seed=5, std=0.06), context=0, prompt=[1, 84, 61, 35, 90, 107, 100, 119], steps=16),
    dict(name="synth_tiny_gelu_tied", synth=dict(shape="tiny", wtype="f16", seed=8, std=0.06, act_type="gelu", tie_word_embeddings=True, rotary_dim=32),
         context=0, prompt=[1, 84, 61, 35, 90, 107, 100, 119], steps=16),
    dict(name="synth_tiny_clip", synth=dict(shape="tiny", wtype="f16", seed=9, std=0.06, qkv_clip=0.5), context=0,
         prompt=[1, 84, 61, 35, 90, 107, 100, 119], steps=16),                                          # a clip that bites (infer.cpp:388-399)
    dict(name="synth_small_f16", synth=dict(shape="small", wtype="f16", seed=1, std=0.03), context=0,
         prompt=[int(t) for t in np.random.default_rng(0).integers(3, 4096, size=40)], steps=12),      # GQA 8:2, head_dim 128
    dict(name="synth_small_f16_T48", synth=dict(shape="small", wtype="f16", seed=1, std=0.03), context=48,
         prompt=[int(t) for t in np.random.default_rng(0).integers(3, 4096, size=60)], steps=12),      # prompt longer than the window
]


def ref_lib():
    L = C.CDLL(os.path.join(ROOT, "oracle", "_ref", "libxalm_ref.so"))
    L.xref_load.restype = C.c_void_p
    L.xref_load.argtypes = [C.c_char_p, C.c_int]
    L.xref_last_error.restype = C.c_char_p
    L.xref_free.argtypes = [C.c_void_p]
    L.xref_config.argtypes = [C.c_void_p, C.c_void_p]
    L.xref_forward.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_void_p]
    L.xref_sample_argmax.argtypes = [C.c_void_p]
    L.xref_sample_prob.argtypes = [C.c_void_p, C.c_int]
    L.xref_sample_prob.restype = C.c_float
    L.xref_kv.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_size_t]
    L.xref_x.argtypes = [C.c_void_p, C.c_void_p]
    return L


def run_case(L, case, path):
    h = L.xref_load(path.encode(), case["context"])
    if not h:
        raise RuntimeError(f"{case['name']}: reference failed to load: {L.xref_last_error().decode()}")
    cfg = (C.c_int * 8)()
    L.xref_config(h, cfg)
    dim, _, head_dim, n_layers, _, n_kv_heads, vocab, max_seq_len = list(cfg)
    lg = np.zeros(vocab, np.float32)
    toks = list(case["prompt"])
    for pos, tok in enumerate(case["prompt"]):
        last = pos + 1 == len(case["prompt"])
        assert L.xref_forward(h, tok, pos, 1 if last else 0, lg.ctypes.data_as(C.c_void_p)) == 0
    logits, probs = [], []
    for _ in range(case["steps"]):
        logits.append(lg.copy())
        nxt = L.xref_sample_argmax(h)
        probs.append(L.xref_sample_prob(h, nxt))
        toks.append(nxt)
        assert L.xref_forward(h, nxt, len(toks) - 1, 1, lg.ctypes.data_as(C.c_void_p)) == 0
    logits.append(lg.copy())
    out = dict(tokens=np.array(toks, np.int32), logits=np.stack(logits), probs=np.array(probs, np.float32),
               config=np.array(list(cfg), np.int32))
    n = max_seq_len * n_kv_heads * head_dim
    # the KV rows no forward pass wrote are uninitialised in the reference (new[] without ()): keep rows [0, min(tokens, window))
    rows = min(len(toks), max_seq_len)
    for l in range(n_layers):
        for which, nm in ((0, "k"), (1, "v")):
            buf = np.zeros(n, np.uint16)
            L.xref_kv(h, l, which, buf.ctypes.data_as(C.c_void_p), n)
            out[f"{nm}_{l}"] = buf[: rows * n_kv_heads * head_dim].copy()
    x = np.zeros(dim, np.float32)
    L.xref_x(h, x.ctypes.data_as(C.c_void_p))
    out["x"] = x
    L.xref_free(h)
    return out


def main():
    L = ref_lib()
    for case in CASES:
        with tempfile.TemporaryDirectory() as td:
            if "file" in case:
                path = os.path.join(HERE, case["file"])
            else:
                path = os.path.join(td, "m.xalm")
                kw = dict(case["synth"])
                synth.write_checkpoint(path, kw.pop("shape"), kw.pop("wtype"), kw.pop("seed"), std=kw.pop("std"), **kw)
            out = run_case(L, case, path)
        meta = {k: v for k, v in case.items()}
        out["case"] = np.frombuffer(json.dumps(meta).encode(), dtype=np.uint8)
        np.savez_compressed(os.path.join(HERE, f"ref_fwd_{case['name']}.npz"), **out)
        print(case["name"], "tokens", out["tokens"][-8:], "logit std %.3f" % out["logits"].std(), flush=True)


if __name__ == "__main__":
    main()
