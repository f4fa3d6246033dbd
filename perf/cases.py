"""Workloads whose speed is watched: what a program does with this framework through xalm_b200.model.Model, from the smallest call to the largest.

Two kinds of model, each with random weights of the layer shapes that the tests and bench.py use:

  llama      Llama / Mistral checkpoints in the weight formats they come in.  "decode": one token at position `ctx` of a filled cache, logits back to
             the host (what a sampler reads).  "prompt": a prompt in one batched pass, the last position's logits.  "score": perplexity mode, every
             position's target probability.
  bolovik, kubolorn, pavitar
             config.json families in the 16-bit serving mode; between them every kind of layer the sequence engine runs often: windowed, chunked and
             sink attention, latent attention, the delta rule, a state-space mixer, gated linear attention, dense and expert feed-forwards.
             "chat": a prompt, then `steps` single tokens whose logits come back one by one, then the sequence is released.  "score": as above.

`exact` restates the models in float64 with plain torch operations.
"""
import json
import math
import zlib

import numpy as np
import torch

from xalm_b200 import capi, synth, types as T, xalm_file as X
from xalm_b200.model import InferenceState, Model

VOCAB = 32000
EPS = 1e-5
HEAD = 128  # head size of every shape here
THETA = 1000000.0
BITS = {"q8_0": 8.5, "q4_0": 4.5, "f16": 16, "bf16": 16, "f8_e4m3": 8}


# ---- the cases ---------------------------------------------------------------------------------------------------------------------------
def llama(name, call, fmt, dim, layers, tokens):
    c = {"model": "llama", "call": call, "format": fmt, "dim": dim, "layers": layers, "tokens": tokens}
    return c if name is None else dict(c, name=name)


def family(name, model, call, width, layers, chunk, prompt, steps):
    c = {"model": model, "call": call, "width": width, "layers": layers, "chunk": chunk, "prompt": prompt, "steps": steps}
    return c if name is None else dict(c, name=name)


def listed():
    return [
        llama("small_q8_0_decode", "decode", "q8_0", 1024, 4, 96),               # a small draft model early in a reply: latency and launches
        llama("7b_q8_0_decode", "decode", "q8_0", 4096, 32, 3001),               # the headline: a 7B model, all layers, deep in its context
        llama("7b_q4_0_decode", "decode", "q4_0", 4096, 8, 700),                 # 4-bit weights, an ordinary context; depth cut
        llama("2048_bf16_decode", "decode", "bf16", 2048, 6, 1777),              # unquantised weights at a middle width, ragged context
        llama("7b_q8_0_score_4096", "score", "q8_0", 4096, 4, 4096),             # perplexity over a full context; depth cut
        llama("7b_f16_prompt_333", "prompt", "f16", 4096, 3, 333),               # an ordinary ragged prompt
        family("bolovik_4096_chat", "bolovik", "chat", 4096, 2, 1024, 1000, 48),  # prompt and reply at the largest width
        family("bolovik_1024_score", "bolovik", "score", 1024, 2, 1024, 2048, 0),  # scoring a text with a small model
        family("kubolorn_1024_chat", "kubolorn", "chat", 1024, 4, 256, 301, 32),  # short ragged prompt, default pass length
        family("kubolorn_2048_prompt", "kubolorn", "chat", 2048, 2, 1024, 2048, 4),  # long prompt, a few tokens of answer
        family("pavitar_2048_chat", "pavitar", "chat", 2048, 2, 256, 777, 48),    # latent and chunked attention, prompt and reply
        family("pavitar_1024_score", "pavitar", "score", 1024, 2, 1024, 1900, 0),  # scoring a ragged text
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["decode", "decode", "prompt", "score", "chat", "chat", "score family"])
    if call in ("decode", "prompt", "score"):
        dim = rng.choice([1024, 2048, 4096])
        fmt = rng.choice(["q8_0", "q8_0", "q4_0", "bf16", "f16", "f8_e4m3"])
        tokens = log_uniform(rng, 24, 4000) if call == "decode" else log_uniform(rng, 33, 2048)
        return llama(None, call, fmt, dim, rng.randint(2, 4), tokens)
    model = rng.choice(["bolovik", "kubolorn", "pavitar"])
    width, chunk = rng.choice([1024, 1024, 1024, 2048]), rng.choice([256, 1024])
    if call == "chat":
        return family(None, model, "chat", width, 2, chunk, log_uniform(rng, 16, 2048), rng.randint(4, 64))
    return family(None, model, "score", width, 2, chunk, log_uniform(rng, 64, 2048), 0)


# ---- models ------------------------------------------------------------------------------------------------------------------------------
def llama_sizes(c):
    dim = c["dim"]
    return dict(dim=dim, hidden_dim={1024: 2816, 2048: 6144, 4096: 14336}[dim], head_dim=HEAD, n_layers=c["layers"], n_heads=dim // HEAD, n_kv_heads=max(2, dim // HEAD // 4),
                vocab_size=VOCAB, max_seq_len=4096, rope_theta=THETA)


def llama_shapes(c):
    z = llama_sizes(c)
    D, F, q, kv = z["dim"], z["hidden_dim"], z["n_heads"] * HEAD, z["n_kv_heads"] * HEAD
    out = {"embed.weight": (VOCAB, D)}
    for i in range(c["layers"]):
        p = f"l.{i}."
        out.update({p + "attn.norm.weight": (D,), p + "attn.q.weight": (q, D), p + "attn.k.weight": (kv, D), p + "attn.v.weight": (kv, D), p + "attn.down.weight": (D, q),
                    p + "mlp.norm.weight": (D,), p + "mlp.gate.weight": (F, D), p + "mlp.down.weight": (D, F), p + "mlp.up.weight": (F, D)})
    out.update({"output.norm.weight": (D,), "output.weight": (VOCAB, D)})
    return out


def family_config(c):
    """bench.py's models: layer kinds alternate; mixtures hold 16 experts of ff / 4 of which 4 are chosen (8 and 2 at width 4096)."""
    W, n = c["width"], c["layers"]
    H, ff, window = W // HEAD, 14336 if W == 4096 else 4 * W, W // 2
    G, rh, rd = H // 4, 4 if W == 1024 else 8, 128 if W == 4096 else 64
    heads = {"heads": H, "kv_heads": G, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5}
    E = 8 if W == 4096 else 16
    expert = {"kind": "moe", "expert": {"ff": ff // 4}}
    out = {"vocab": VOCAB, "width": W, "norm": {"eps": EPS}}
    if c["model"] == "bolovik":
        att = dict(heads, mask={"size": window, "keep_first": 64}, rot={"base": 10000.0, "dims": HEAD // 2})
        delta = {"heads": 2 * rh, "kv_heads": rh, "dim": rd, "vdim": HEAD, "conv": 4}
        moe = dict(expert, router={"experts": E, "top": E // 4, "groups": {"count": 4, "keep": 2}})
        pair = [{"type": "attention", "mixer": att, "mlp": {"kind": "dense", "ff": ff}}, {"type": "delta", "mixer": delta, "mlp": moe}]
        out.update(architecture="Bolovik", norm={"eps": EPS, "groups": 8})
    elif c["model"] == "kubolorn":
        att = dict(heads, rot={"base": 10000.0, "dims": HEAD // 2})
        ssd = {"heads": 2 * rh, "vdim": HEAD, "state": rd, "groups": rh, "conv": 4, "norm_groups": 4}
        gla = {"heads": 2 * rh, "dim": rd, "vdim": HEAD, "tau": 8.0}
        moe = dict(expert, router={"experts": E, "top": E // 4})
        pair = [{"type": "parallel", "mixer": {"left": att, "right": ssd, "left_scale": 1.0, "right_scale": 0.7}, "mlp": {"kind": "dense", "ff": ff}},
                {"type": "gla", "mixer": gla, "mlp": moe}]
        out.update(architecture="Kubolorn", norm={"eps": EPS, "groups": 8}, canon={"taps": 4},
                   embedding={"scale": float(W) ** 0.5, "bigram": {"buckets": 8191, "mul_prev": 1000003, "mul_cur": 7919}})
    else:
        lat = {"heads": H, "dim": HEAD, "vdim": HEAD, "kv_rank": min(512, max(256, W // 4)), "q_rank": 3 * W // 8, "scale": HEAD ** -0.5, "mask": {"size": window}}
        att = dict(heads, mask={"size": window}, rot={"base": 10000.0, "dims": HEAD // 2})
        moe = dict(expert, router={"experts": E, "top": E // 4}, shared={"ff": ff // 4})
        pair = [{"type": "latent_attention", "mixer": lat, "mlp": moe}, {"type": "attention", "mixer": att, "mlp": moe}]
        out.update(architecture="Pavitar", logit_softcap=30.0)
    out["layers"] = (pair * n)[:n]
    return out


def family_shapes(cfg):
    """Every tensor of the model by name.  For the bench shapes the decay's inner size of a gated-linear-attention layer is 32."""
    W, kind = cfg["width"], cfg["architecture"]
    out = {"embed": (VOCAB, W), "final.norm": (W,)}
    if kind == "Bolovik":
        out["head"] = (VOCAB, W)
    if kind == "Kubolorn":
        out.update({"bigram": (cfg["embedding"]["bigram"]["buckets"] + 1, W), "embed.norm": (W,)})
    for i, L in enumerate(cfg["layers"]):
        p, m, mx, mlp = f"l{i}.", f"l{i}.mix.", L["mixer"], L["mlp"]
        out.update({p + "norm1": (W,), p + "norm2": (W,)})
        if kind == "Kubolorn":
            out.update({p + "canon1": (W, 4), p + "canon2": (W, 4)})
        if L["type"] == "parallel":
            a, b = mx["left"], mx["right"]
            inner, gn = b["heads"] * b["vdim"], b["groups"] * b["state"]
            out.update({m + "left.q": (a["heads"] * HEAD, W), m + "left.k": (a["kv_heads"] * HEAD, W), m + "left.sink": (a["heads"],), m + "left.o": (W, a["heads"] * HEAD),
                        m + "right.in": (2 * inner + 2 * gn + b["heads"], W), m + "right.conv": (inner + 2 * gn, 4), m + "right.conv.b": (inner + 2 * gn,),
                        m + "right.norm": (inner,), m + "right.o": (W, inner), **{m + "right." + k: (b["heads"],) for k in ("dt_bias", "A_log", "D")}})
        elif L["type"] == "latent_attention":
            H, R, Rq = mx["heads"], mx["kv_rank"], mx["q_rank"]
            out.update({m + "dq": (Rq, W), m + "dq.norm": (Rq,), m + "uq": (H * HEAD, Rq), m + "dkv": (R, W), m + "dkv.norm": (R,), m + "uk": (H * HEAD, R),
                        m + "uv": (H * HEAD, R), m + "g": (H, W), m + "o": (W, H * HEAD)})
        else:
            H, G, d, dv = mx["heads"], mx.get("kv_heads", mx["heads"]), mx["dim"], mx["vdim"]
            delta, gla = L["type"] == "delta", L["type"] == "gla"
            out.update({m + "q": ((G if delta else H) * d, W), m + "k": (G * d, W), m + "v": ((H if delta or gla else G) * dv, W), m + "o": (W, H * dv)})
            if delta:
                out.update({m + "q.conv": (G * d, 4), m + "k.conv": (G * d, 4), m + "v.conv": (H * dv, 4), m + "b": (H, W), m + "a": (H, W), m + "g": (H * dv, W),
                            m + "A_log": (H,), m + "dt_bias": (H,), m + "norm": (dv,)})
            elif gla:
                out.update({m + "g": (H * dv, W), m + "norm": (dv,), m + "a1": (32, W), m + "a2": (H * d, 32), m + "a2.b": (H * d,)})
            elif kind == "Pavitar":
                out.update({m + "q.norm": (H * d,), m + "k.norm": (G * d,)})
        if mlp["kind"] == "dense":
            parts, extra = {"": mlp["ff"]}, {}
        else:
            E = mlp["router"]["experts"]
            parts = {f"e{e}.": mlp["expert"]["ff"] for e in range(E)}
            extra = {"router": (E, W)}
            if kind == "Pavitar":
                parts["shared."] = mlp["shared"]["ff"]
                extra.update({"router.b": (E,), "shared.sg": (1, W)})
        for s, ff in parts.items():
            out.update({p + "mlp." + s + "up": (ff, W), p + "mlp." + s + "down": (W, ff)})
            if kind != "Kubolorn":
                out[p + "mlp." + s + "gate"] = (ff, W)
        out.update({p + "mlp." + k: v for k, v in extra.items()})
    return out


def generator(seed, name):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
    return g


def normal(seed, name, shape):
    return torch.randn(shape, generator=generator(seed, name), device="cuda", dtype=torch.float32)


def llama_source(name):
    """Layer i holds the same values as layer i + 4, which keeps making a deep model quick; every layer has its own copy on the device."""
    part = name.split(".")
    return ".".join([part[0], str(int(part[1]) % 4)] + part[2:]) if part[0] == "l" else name


def llama_weight(c, seed, name, shape):
    """(framework type, stored bytes, values as float64 on demand): rows of standard deviation 1.28 / sqrt(columns)."""
    if len(shape) == 1:
        w = 1.0 + 0.1 * normal(seed, name, shape)
        return T.F32, w, w.double
    std = 1.28 / math.sqrt(shape[1])
    w = normal(seed, name, shape)
    if c["format"] in ("f16", "bf16"):
        w = (std * w).to(torch.float16 if c["format"] == "f16" else torch.bfloat16)
        return T.parse(c["format"]), w, w.double
    if c["format"] == "f8_e4m3":
        w = (std * w).to(torch.float8_e4m3fn)
        return T.F8_E4M3, w, lambda: w.float().double()
    # blocks of 32: a 16-bit step and the whole numbers it multiplies
    top = 127 if c["format"] == "q8_0" else 7
    w = w.view(shape[0], shape[1] // 32, 32)
    step = (w.abs().amax(-1, keepdim=True) * (std / top)).half()
    q = (w * std / step.float()).round_().clamp_(-top, top)
    if c["format"] == "q8_0":
        raw = torch.cat([step.view(torch.uint8), q.to(torch.int8).view(torch.uint8)], -1)
    else:
        u = (q + 8).to(torch.uint8)
        raw = torch.cat([step.view(torch.uint8), u[..., :16] | (u[..., 16:] << 4)], -1)
    return T.parse(c["format"]), raw, lambda: (step.double() * q.double()).view(shape)


def family_weight(seed, name, shape):
    """bfloat16, spread as bench.py spreads them."""
    leaf, w = name.split(".")[-1], normal(seed, name, shape)
    if leaf in ("conv", "canon1", "canon2"):
        w = 0.4 * w
    elif name == "embed" and len(shape) == 2:
        w = w / math.sqrt(shape[1])
    elif len(shape) == 2:
        w = w * ((2.0 if leaf == "router" else 1.0) / math.sqrt(shape[1]))
    elif leaf == "A_log":
        w = -1.5 + 0.8 * w.clamp(-2, 2)
    elif leaf in ("sink", "dt_bias") or name.endswith("conv.b"):
        w = 0.2 * w
    elif leaf == "b":
        w = 3.0 + w if name.endswith("a2.b") else 0.1 * w
    elif leaf in ("norm1", "norm2"):
        w = 0.3 + 0.05 * w
    else:
        w = 1.0 + 0.1 * w
    return w.to(torch.bfloat16)





def host_bytes(t):
    return t.contiguous().view(torch.uint8).reshape(-1).cpu().numpy()


def token_ids(seed, n):
    return torch.randint(3, VOCAB, (n,), generator=generator(seed, "tokens"), device="cuda").cpu().numpy().astype(np.int32)


def prepare(case, seed):
    if case["model"] == "llama":
        cfg = X.parse_config(synth.metadata_strings(synth.model_config("m7", **llama_sizes(case))), 4096)
        tensors, made = {}, {}
        for name, shape in llama_shapes(case).items():
            src = llama_source(name)
            if src not in made:
                kind, raw, _ = llama_weight(case, seed, src, shape)
                made[src] = (kind, shape, host_bytes(raw))
            tensors[name] = made[src]
        model = Model(cfg, tensors).cuda(release_host=True)
        ids = token_ids(seed, case["tokens"] + 1)
        if case["call"] == "decode":
            model.prefill(ids[:-1], 0, want_logits=0)
        return {"call": case["call"], "model": model, "ids": ids, "state": InferenceState(cfg).cuda()}
    cfg = family_config(case)
    tensors = {n: (T.BF16, s, host_bytes(family_weight(seed, n, s))) for n, s in family_shapes(cfg).items()}
    capi.tune("seq_chunk", case["chunk"])
    model = Model({"architecture": cfg["architecture"], "json": json.dumps(cfg), "vocab_size": VOCAB}, tensors).cuda(max_tokens=case["prompt"] + case["steps"])
    capi.tune("seq_chunk", 256)
    model.tensors.clear()
    state = {"call": case["call"] + " family", "model": model, "ids": token_ids(seed, case["prompt"] + max(1, case["steps"])), "prompt": case["prompt"],
             "state": InferenceState(model.config).cuda()}
    if case["call"] == "chat":
        state["logits"] = np.zeros((case["steps"] + 1, VOCAB), dtype=np.float32)
    return state


def run(s):
    model, ids, call = s["model"], s["ids"], s["call"]
    if call == "decode":
        model.forward(s["state"], int(ids[-1]), len(ids) - 1)
        return s["state"].logits()
    if call == "prompt":
        return model.prefill(ids[:-1], 0, want_logits=1)
    if call == "score":
        return model.prefill(ids[:-1], 0, want_logits=2, targets=ids[1:], fetch_logits=False)[1]
    model.release()
    n = s["prompt"]
    if call == "score family":
        return model.prefill(ids[:n], 0, want_logits=2, targets=ids[1:n + 1], fetch_logits=False)[1]
    out = s["logits"]
    out[0] = model.prefill(ids[:n], 0, want_logits=1)
    for i in range(len(out) - 1):  # the reply's tokens are given, so that every step's logits can be compared
        model.forward(s["state"], int(ids[n + i]), n + i)
        out[i + 1] = s["state"].logits()
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------------------
def seen(n, window):
    """Pairs of positions of a causal window over positions 0 .. n - 1."""
    w = min(n, window)
    return w * (w + 1) // 2 + (n - w) * w


def work(case):
    if case["model"] == "llama":
        z, n = llama_sizes(case), case["tokens"]
        D, kv, L = z["dim"], z["n_kv_heads"] * HEAD, case["layers"]
        layer = 2 * D * D + 2 * D * kv + 3 * D * z["hidden_dim"]
        weights = L * layer + VOCAB * D
        if case["call"] == "decode":
            return {"bytes": weights * BITS[case["format"]] / 8 + L * 4 * kv * (n + 1) + 4 * VOCAB, "flops": 2 * weights + 4 * L * D * (n + 1)}
        rows = n if case["call"] == "score" else 1
        return {"bytes": weights * BITS[case["format"]] / 8 + L * 4 * kv * n + 4 * (n if rows > 1 else VOCAB),
                "flops": 2 * (L * layer * n + VOCAB * D * rows) + 4 * L * D * seen(n, n)}
    cfg = family_config(case)
    n, steps, H = case["prompt"], case["steps"], case["width"] // HEAD
    every = active = state = cache = 0
    flops = 0
    total = n + steps
    for name, shape in family_shapes(cfg).items():
        if len(shape) == 2 and name not in ("embed", "head", "bigram"):
            every += shape[0] * shape[1]
            active += shape[0] * shape[1] * (0.25 if ".mlp.e" in name else 1)
    for L in cfg["layers"]:
        mx = L["mixer"]
        for m in ((mx["left"], mx["right"]) if L["type"] == "parallel" else (mx,)):
            if L["type"] in ("delta", "gla") or "state" in m:
                s = m["heads"] * m.get("dim", m.get("state")) * m["vdim"]
                state += 2 * 4 * s
                flops += (6 if L["type"] == "delta" else 4) * s * total
            else:
                pairs = seen(total, m["mask"]["size"] if "mask" in m else total)
                flops += 4 * HEAD * H * pairs
                row = m["kv_rank"] if L["type"] == "latent_attention" else 2 * m["kv_heads"] * HEAD
                cache += 2 * row * (n + steps * min(total, m["mask"]["size"] if "mask" in m else total))
    head = VOCAB * case["width"]
    rows = n if case["call"] == "score" else 1 + steps
    return {"bytes": 2 * (every + head) + steps * (2 * (active + head) + state) + cache + 4 * (n if case["call"] == "score" else rows * VOCAB),
            "flops": flops + 2 * active * total + 2 * head * rows}


def tolerance(case):
    # Distances from float64 as measured: Llama 1e-3 (2e-3 at 32 layers: 16-bit cache, batched passes with operands of 22 bits), bolovik and pavitar 4e-3
    # to 4e-2 (products with 16-bit operands; a token whose two closest experts change places differs in its own row only), kubolorn 1e-4 (its tied
    # head returns the token's own embedding as the largest logit).
    if case["model"] == "llama":
        return {"rel": 6e-3, "max": 6e-2}
    return {"rel": 2e-3, "max": 0.3} if case["model"] == "kubolorn" else {"rel": 2e-2, "max": 0.9}


# ---- float64 -----------------------------------------------------------------------------------------------------------------------------
def unit(x, eps=EPS):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()


def group_unit(x, groups):
    return unit(x.unflatten(-1, (groups, -1))).flatten(-2)


def silu(x):
    return x * torch.sigmoid(x)


def gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def turn(x, freq, neighbours, mag=1.0):
    """x (n, heads, d): the first 2 len(freq) entries of every head, turned by position times frequency."""
    r = len(freq)
    a = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None] * freq
    c, s = (a.cos() * mag)[:, None], (a.sin() * mag)[:, None]
    out = x.clone()
    i, j = (slice(0, 2 * r, 2), slice(1, 2 * r, 2)) if neighbours else (slice(0, r), slice(r, 2 * r))
    out[..., i], out[..., j] = x[..., i] * c - x[..., j] * s, x[..., j] * c + x[..., i] * s
    return out


def frequencies(base, dims):
    return base ** (-2.0 * torch.arange(dims // 2, device="cuda", dtype=torch.float64) / dims)


def attend(q, k, v, scale, mask, sink=None):
    """q (n, H, d), k (n, G, d), v (n, G, dv); mask (n, n) True where seen.  Returns (n, H dv)."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T * scale).masked_fill_(~mask, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        out.append(torch.softmax(s, 1)[:, :n] @ v[:, h * G // H])
    return torch.cat(out, 1)


def conv(x, w, bias=None):
    """Causal depthwise convolution over the rows; the last column of w multiplies the current one."""
    taps = w.shape[1]
    ext = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(ext[j:j + x.shape[0]] * w[:, j] for j in range(taps))
    return y if bias is None else y + bias


def exact_llama(case, seed):
    z, shapes, n = llama_sizes(case), llama_shapes(case), case["tokens"] + (case["call"] == "decode")
    H, G = z["n_heads"], z["n_kv_heads"]
    ids = torch.from_numpy(token_ids(seed, case["tokens"] + 1)).cuda().long()

    def w(name):
        return llama_weight(case, seed, llama_source(name), shapes[name])[2]()

    pos = torch.arange(n, device="cuda")
    mask, freq = pos[:, None] >= pos, frequencies(THETA, HEAD)
    x = w("embed.weight")[ids[:n]]
    for i in range(case["layers"]):
        p = f"l.{i}."
        h = unit(x) * w(p + "attn.norm.weight")
        q, k, v = ((h @ w(p + f"attn.{m}.weight").T).view(n, -1, HEAD) for m in "qkv")
        assert q.shape[1] == H and k.shape[1] == G
        x = x + attend(turn(q, freq, True), turn(k, freq, True), v, HEAD ** -0.5, mask) @ w(p + "attn.down.weight").T
        h = unit(x) * w(p + "mlp.norm.weight")
        x = x + (silu(h @ w(p + "mlp.gate.weight").T) * (h @ w(p + "mlp.up.weight").T)) @ w(p + "mlp.down.weight").T
    if case["call"] != "score":
        x = x[-1:]
    logits = (unit(x) * w("output.norm.weight")) @ w("output.weight").T
    if case["call"] == "score":
        return torch.softmax(logits, 1).gather(1, ids[1:n + 1, None])[:, 0]
    return logits[0]


def delta_mixer(x, w, m, mx):
    H, G, d, dv, n = mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"], x.shape[0]
    q, k, v = (silu(conv(x @ w(m + c).T, w(m + c + ".conv"))) for c in "qkv")
    q, k = ((a / (a.square().sum(-1, keepdim=True) + 1e-6).sqrt()).repeat_interleave(H // G, 1) for a in (q.view(n, G, d), k.view(n, G, d)))
    v, q = v.view(n, H, dv), q * d ** -0.5
    beta = torch.sigmoid(x @ w(m + "b").T)
    decay = torch.exp(-w(m + "A_log").exp() * torch.nn.functional.softplus(x @ w(m + "a").T + w(m + "dt_bias"), threshold=1e9))
    S, out = x.new_zeros(H, d, dv), []
    for t in range(n):
        S = decay[t, :, None, None] * S
        u = beta[t, :, None] * (v[t] - torch.einsum("hij,hi->hj", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None]
        out.append(torch.einsum("hij,hi->hj", S, q[t]))
    o = unit(torch.stack(out)) * w(m + "norm")
    return (o.reshape(n, H * dv) * silu(x @ w(m + "g").T)) @ w(m + "o").T


def keyed(q, k, v, f, s):
    """S <- f S + s k v^T, o = S^T q per head, f (n, H, d)."""
    S, out = q.new_zeros(v.shape[1], q.shape[2], v.shape[2]), []
    for t in range(q.shape[0]):
        S = f[t, :, :, None] * S + (s[t] * k[t])[:, :, None] * v[t, :, None]
        out.append(torch.einsum("hij,hi->hj", S, q[t]))
    return torch.stack(out)


def ssd_mixer(h, w, m, mx):
    H, P, N, G, n = mx["heads"], mx["vdim"], mx["state"], mx["groups"], h.shape[0]
    inner, u = H * P, h @ w(m + "in").T
    z, xbc, dt = u.split([inner, inner + 2 * G * N, H], 1)
    x, B, C = silu(conv(xbc, w(m + "conv"), w(m + "conv.b"))).split([inner, G * N, G * N], 1)
    x, B, C = x.view(n, H, P), *(a.view(n, G, N).repeat_interleave(H // G, 1) for a in (B, C))
    dt = torch.nn.functional.softplus(dt + w(m + "dt_bias"), threshold=1e9)[:, :, None]
    y = keyed(C, B, x, torch.exp(-w(m + "A_log").exp()[:, None] * dt).expand(n, H, N), dt) + w(m + "D")[:, None] * x
    return (group_unit(y.reshape(n, inner) * silu(z), mx["norm_groups"]) * w(m + "norm")) @ w(m + "o").T


def gla_mixer(h, w, m, mx):
    H, d, dv, n = mx["heads"], mx["dim"], mx["vdim"], h.shape[0]
    q, k, v = (h @ w(m + "q").T).view(n, H, d) * d ** -0.5, (h @ w(m + "k").T).view(n, H, d), (h @ w(m + "v").T).view(n, H, dv)
    f = torch.sigmoid((h @ w(m + "a1").T) @ w(m + "a2").T + w(m + "a2.b")) ** (1.0 / mx["tau"])
    o = unit(keyed(q, k, v, f.view(n, H, d), torch.ones(n, 1, 1, device="cuda", dtype=torch.float64))) * w(m + "norm")
    return (o.reshape(n, H * dv) * silu(h @ w(m + "g").T)) @ w(m + "o").T


def gated(h, w, p, act=silu):
    return (act(h @ w(p + "gate").T) * (h @ w(p + "up").T)) @ w(p + "down").T


def mixture(h, w, p, expert, score, top, allowed=None):
    """Sum over the `top` experts of the largest scores; score -> weights of the chosen."""
    s, weights = score
    idx = (s if allowed is None else s.masked_fill(~allowed, -math.inf)).topk(top, 1).indices
    wgt, out = weights(s.gather(1, idx)), torch.zeros_like(h)
    for e in range(s.shape[1]):
        t, slot = (idx == e).nonzero(as_tuple=True)
        if len(t):
            out[t] += wgt[t, slot, None] * expert(h[t], p + f"e{e}.")
    return out


def exact_family(case, seed):
    cfg = family_config(case)
    shapes, kind, groups = family_shapes(cfg), cfg["architecture"], cfg["norm"].get("groups", 1)

    def w(name):
        return family_weight(seed, name, shapes[name]).double()

    n = case["prompt"] + case["steps"]
    ids = torch.from_numpy(token_ids(seed, case["prompt"] + max(1, case["steps"]))).cuda().long()
    pos = torch.arange(n, device="cuda")
    causal = pos[:, None] >= pos
    x = w("embed")[ids[:n]]
    if kind == "Kubolorn":
        bg = cfg["embedding"]["bigram"]
        pair = (ids[:n - 1] * bg["mul_prev"] + ids[1:n] * bg["mul_cur"]) % bg["buckets"]
        x = x * cfg["embedding"]["scale"] + w("bigram")[torch.cat([torch.full((1,), bg["buckets"], device="cuda"), pair])]
        x = group_unit(x, groups) * w("embed.norm")
    for i, L in enumerate(cfg["layers"]):
        p, m, mx = f"l{i}.", f"l{i}.mix.", L["mixer"]
        freq, top = frequencies(10000.0, HEAD // 2), L["mlp"].get("router", {}).get("top")
        if kind == "Bolovik":
            if L["type"] == "attention":
                q, k, v = ((x @ w(m + c).T).view(n, -1, HEAD) for c in "qkv")
                mask = causal & ((pos[:, None] - pos < mx["mask"]["size"]) | (pos < mx["mask"]["keep_first"]))
                y = attend(unit(turn(q, freq, False)), unit(turn(k, freq, False)), unit(v), mx["scale"], mask) @ w(m + "o").T
            else:
                y = delta_mixer(x, w, m, mx)
            x = x + group_unit(y, groups) * w(p + "norm1")
            if L["mlp"]["kind"] == "dense":
                y = gated(x, w, p + "mlp.", gelu)
            else:
                s = torch.sigmoid(x @ w(p + "mlp.router").T)
                best = s.view(n, 4, -1).topk(2, 2).values.sum(2).topk(2, 1).indices
                allowed = torch.zeros(n, 4, device="cuda", dtype=torch.bool).scatter_(1, best, True).repeat_interleave(s.shape[1] // 4, 1)
                y = mixture(x, w, p + "mlp.", lambda h, q: gated(h, w, q), (s, lambda g: g), top, allowed)
            x = x + group_unit(y, groups) * w(p + "norm2")
        elif kind == "Kubolorn":
            def read(a, b):
                h = group_unit(x, groups) * w(p + a)
                return h + conv(h, w(p + b))
            h1, h2 = read("norm1", "canon1"), read("norm2", "canon2")
            if L["type"] == "parallel":
                k = (h1 @ w(m + "left.k").T).view(n, -1, HEAD)
                q = (h1 @ w(m + "left.q").T).view(n, -1, HEAD)
                a = attend(turn(q, freq, False), turn(k, freq, False), k, HEAD ** -0.5, causal, w(m + "left.sink")) @ w(m + "left.o").T
                y = mx["left_scale"] * a + mx["right_scale"] * ssd_mixer(h1, w, m + "right.", mx["right"])
            else:
                y = gla_mixer(h1, w, m, mx)
            if L["mlp"]["kind"] == "dense":
                y = y + gelu(h2 @ w(p + "mlp.up").T) @ w(p + "mlp.down").T
            else:
                y = y + mixture(h2, w, p + "mlp.", lambda h, q: (h @ w(q + "up").T).clamp(min=0).square() @ w(q + "down").T,
                                (h2 @ w(p + "mlp.router").T, lambda g: torch.softmax(g, 1)), top)
            x = x + y
        else:
            h, size = unit(x) * (1.0 + w(p + "norm1")), mx["mask"]["size"]
            if L["type"] == "latent_attention":
                q = (unit(h @ w(m + "dq").T) * w(m + "dq.norm")) @ w(m + "uq").T
                c = unit(h @ w(m + "dkv").T) * w(m + "dkv.norm")
                o = attend(q.view(n, -1, HEAD), (c @ w(m + "uk").T).view(n, -1, HEAD), (c @ w(m + "uv").T).view(n, -1, HEAD), mx["scale"], causal & (pos[:, None] - pos < size))
                o = (o.view(n, -1, HEAD) * torch.sigmoid(h @ w(m + "g").T)[:, :, None]).view(n, -1)
            else:
                q, k, v = unit(h @ w(m + "q").T) * w(m + "q.norm"), unit(h @ w(m + "k").T) * w(m + "k.norm"), h @ w(m + "v").T
                q, k, v = turn(q.view(n, -1, HEAD), freq, True), turn(k.view(n, -1, HEAD), freq, True), v.view(n, -1, HEAD)
                o = attend(q, k, v, mx["scale"], causal & (pos[:, None] // size == pos // size))
            x = x + o @ w(m + "o").T
            h = unit(x) * (1.0 + w(p + "norm2"))
            y = mixture(h, w, p + "mlp.", lambda a, q: gated(a, w, q), (h @ w(p + "mlp.router").T + w(p + "mlp.router.b"), lambda g: torch.softmax(g, 1)), top)
            x = x + y + torch.sigmoid(h @ w(p + "mlp.shared.sg").T) * gated(h, w, p + "mlp.shared.")
    if case["call"] == "chat":
        x = x[case["prompt"] - 1:]
    if kind == "Bolovik":
        logits = (group_unit(x, groups) * w("final.norm")) @ w("head").T
    else:
        logits = (group_unit(x, groups) * (w("final.norm") + (kind == "Pavitar"))) @ w("embed").T
    if "logit_softcap" in cfg:
        logits = cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])
    if case["call"] == "score":
        return torch.softmax(logits, 1).gather(1, ids[1:n + 1, None])[:, 0]
    return logits


def exact(case, seed):
    return exact_llama(case, seed) if case["model"] == "llama" else exact_family(case, seed)
