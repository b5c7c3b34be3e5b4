"""The work this library is measured on: requests of token ids through ``Engine.step``.

A case is a batch of requests: the prompts run in one step, then every sequence advances by one given
token per captured decode step, and all logits come back.  (The decoded tokens are given, not sampled, so
that two runs see the same inputs whatever the last bit of a logit is.)  Weights are random, with the sizes
of the configurations that ``bench.py`` and the tests use and fewer layers than the full models where those
have dozens: a layer costs the same in any number of them, and rounding has fewer layers to add up over.

``exact`` restates each decoder in plain torch, in 64 bits, a sequence at a time.
"""
import math
import random
import re

import torch

from rbitnet_b200 import Engine, StepEntry
from rbitnet_b200.config import config_from_dict, get_architecture

VOCAB = 32000


# ------------------------------------------------------------------------------------------- the models
def _llama(width, heads, kv, dim, ff, layers, vocab, theta, eps, positions):
    return {"architectures": ["LlamaForCausalLM"], "num_hidden_layers": layers, "hidden_size": width,
            "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": dim, "intermediate_size": ff,
            "vocab_size": vocab, "rope_theta": theta, "rms_norm_eps": eps, "max_position_embeddings": positions,
            "tie_word_embeddings": False, "hidden_act": "silu"}


def _design(name, layers, **more):
    return {"architecture": name, "vocab": VOCAB, "width": 2048, "norm": {"eps": 1e-6}, "max_positions": 8192,
            "layers": layers, **more}


def _safuvik():
    left = {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 64, "scale": 128 ** -0.5, "mask": {"size": 1024},
            "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}}
    mlp = {"kind": "dense", "ff": 5632, "limit": 7.0}
    par = {"type": "parallel", "mlp": mlp, "mixer": {"left": left, "right": {"width": 2048, "blocks": 16, "conv": 4}}}
    mem = {"type": "mlstm", "mlp": mlp, "mixer": {"heads": 8, "dim": 128, "vdim": 256, "gate_cap": 15.0}}
    return _design("Safuvik", [par, par, mem, par, par, mem], streams=4, logit_scale=1.0)


def _vaderax():
    att = {"type": "attention", "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                                          "rot": {"base": 10000.0, "dims": 64}}}
    delta = {"type": "delta", "mixer": {"heads": 16, "kv_heads": 8, "dim": 128, "vdim": 128, "conv": 4}}
    moe = {"kind": "moe", "expert": {"ff": 1408}, "router": {"experts": 30, "identity": 2, "top": 4,
                                                             "groups": {"count": 8, "keep": 4}}}
    return _design("Vaderax", [dict(delta, mlp={"kind": "dense", "ff": 5632}), dict(delta, mlp=moe), dict(att, mlp=moe),
                               dict(delta, mlp=moe)], embedding={"scale": 1.0}, loop={"start": 1, "stop": 3, "times": 2})


def _nifarax():
    moe = {"kind": "moe", "expert": {"ff": 1408, "limit": 7.0}, "router": {"experts": 32, "top": 4},
           "shared": {"ff": 1408, "limit": 7.0}}
    mem = {"type": "gla", "mlp": moe, "mixer": {"heads": 8, "dim": 128, "vdim": 256, "tau": 16.0, "decay_rank": 16}}
    att = {"type": "latent_attention", "mlp": moe, "mixer": {"heads": 16, "dim": 128, "vdim": 128, "q_rank": 768,
                                                             "kv_rank": 128, "scale": 128 ** -0.5}}
    return _design("Nifarax", [mem, att, att, dict(mem, weights_of=0), att, att], norm={"eps": 1e-6, "groups": 2},
                   canon={"taps": 4}, logit_softcap=30.0)


def _gozotar():
    mlp = {"kind": "dense", "ff": 5632}
    lat = {"type": "latent_attention", "mlp": mlp, "mixer": {
        "heads": 16, "dim": 128, "rot_dim": 32, "vdim": 128, "kv_rank": 96, "scale": 160 ** -0.5,
        "rot": {"base": 10000.0, "dims": 32}}}
    att = {"type": "attention", "mlp": mlp, "mixer": {
        "heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 50.0, "v_mix": True,
        "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
    par = {"type": "parallel", "mlp": mlp, "mixer": {
        "left": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "conv": 4,
                 "rot": {"base": 10000.0, "dims": 64}},
        "right": {"heads": 8, "dim": 128, "vdim": 256, "rot": {"base": 10000.0, "dims": 128},
                  "decay": [1.0 - 2.0 ** (-5 - 3 * i / 7) for i in range(8)]},
        "left_scale": 0.5, "right_scale": 0.5}}
    return _design("Gozotar", [lat, att, par, lat, att, par], token_side={"dim": 256},
                   embedding={"bigram": {"buckets": 100003, "mul_prev": 36313, "mul_cur": 27191}})


def _busavik():
    moe = {"kind": "moe", "expert": {"ff": 1408}, "router": {"experts": 32, "top": 4}, "shared": {"ff": 1408}}
    mixer = {"heads": 16, "dim": 128, "rot_dim": 32, "vdim": 128, "q_rank": 768, "kv_rank": 96, "scale": 160 ** -0.5,
             "rot": {"base": 10000.0, "dims": 32, "scaling": {"factor": 8.0, "original": 2048, "fast": 16.0, "slow": 2.0}}}
    return _design("Busavik", [{"type": "latent_attention", "mixer": mixer, "mlp": m}
                               for m in ({"kind": "dense", "ff": 5632}, moe, {"kind": "dense", "ff": 5632}, moe)],
                   logit_scale=1.0, loop={"start": 1, "stop": 3, "times": 2})


def _bafulorn():
    ssm = {"type": "mamba2", "mixer": {"heads": 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4, "norm_groups": 8}}
    lat = {"type": "latent_attention", "mixer": {"heads": 16, "dim": 128, "vdim": 128, "kv_rank": 128,
                                                 "scale": 128 ** -0.5, "mask": {"size": 1024}}}
    att = {"type": "attention", "mixer": {
        "heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024, "keep_first": 64},
        "rot": {"base": 500000.0, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
    moe = {"kind": "moe", "expert": {"ff": 1408}, "router": {"experts": 32, "top": 4, "scale": 2.5}, "shared": {"ff": 1408}}
    dense = {"kind": "dense", "ff": 5632}
    return _design("Bafulorn", [dict((ssm, lat, att)[i % 3], mlp=moe if i % 2 else dense) for i in range(6)],
                   residual_mult=0.5)


MODELS = {
    # the second of the two tiny configurations the tests run on (one kv head, heads of 32)
    "llama_tiny": lambda: _llama(96, 3, 1, 32, 256, 3, 384, 500000.0, 1e-6, 256),
    "llama_3_8b": lambda: _llama(4096, 32, 8, 128, 14336, 4, 128256, 500000.0, 1e-5, 8192),
    "llama_2_7b": lambda: _llama(4096, 32, 32, 128, 11008, 4, VOCAB, 10000.0, 1e-5, 4096),
    "tinyllama_1b": lambda: _llama(2048, 32, 4, 64, 5632, 6, VOCAB, 10000.0, 1e-5, 2048),
    # the other six architectures at the sizes of bench.py --design ..._w2048
    "safuvik": _safuvik, "vaderax": _vaderax, "nifarax": _nifarax,
    "gozotar": _gozotar, "busavik": _busavik, "bafulorn": _bafulorn,
}


def listed():
    def case(name, model, dtype, batch, shortest, longest, steps):
        return {"name": name, "model": model, "dtype": dtype, "batch": batch, "shortest": shortest, "longest": longest,
                "steps": steps}
    return [
        # the smallest call: a toy model for bring-up in 32 bits, four short prompts, twelve steps; latency and launches
        case("llama tiny f32", "llama_tiny", "float32", 4, 1, 17, 12),
        # the headline: a handful of chat requests on the 8B shape, most of the time in memory-bound decode steps
        case("llama 8b decode b8", "llama_3_8b", "bfloat16", 8, 512, 512, 32),
        # a server's full batch on a small model: launch-bound layers, 64 rows a product
        case("tinyllama decode b64", "tinyllama_1b", "bfloat16", 64, 64, 128, 24),
        # time to the first token of one long prompt on the 8B shape: tensor-core products and attention
        case("llama 8b prefill 2048", "llama_3_8b", "bfloat16", 1, 2048, 2048, 0),
        # a batch job's unequal prompts at once on the 7B shape (as many kv heads as heads); the largest case
        case("llama 7b ragged prefill", "llama_2_7b", "bfloat16", 16, 64, 2048, 0),
        # the 32-bit path at real layer sizes: unequal prompts, then a few steps, as a comparison of logits runs it
        case("tinyllama f32", "tinyllama_1b", "float32", 3, 37, 300, 8),
        # one long prompt through window attention, a gated recurrence and matrix memories
        case("safuvik prefill", "safuvik", "bfloat16", 1, 2048, 2048, 0),
        # two unequal prompts and a short answer: delta rule, routed experts, looped layers
        case("vaderax request", "vaderax", "bfloat16", 2, 501, 1499, 8),
        # eight short requests, most of the time in decode steps: gated linear attention, latents, routed experts
        case("nifarax decode b8", "nifarax", "bfloat16", 8, 128, 128, 32),
        # one prompt of an odd length and a short answer: prepared q and k, sinks, retention, pair embedding
        case("gozotar request", "gozotar", "bfloat16", 1, 1901, 1901, 8),
        # four very unequal prompts and a short answer: latents for queries and keys, tanh norms, routed experts
        case("busavik request", "busavik", "bfloat16", 4, 33, 777, 16),
        # one prompt beyond the attention's window and a short answer: state space, windows with kept positions
        case("bafulorn long prompt", "bafulorn", "bfloat16", 1, 3001, 3001, 16),
    ]


def _cost(case):
    """A rough time in seconds, to keep drawn cases below the largest listed one."""
    w = work(case)
    return w["flops"] / (3e13 if case["dtype"] == "float32" else 8e14) + w["bytes"] / 6e12


def draw(rng):
    """Any model, 1 to 64 sequences, prompts of 1 to 4,096 tokens (equal or not), 0 to 32 decode steps.  (Safuvik: up to 3
    sequences.  With more, its results vary from one run to the next as this file is written: blocks that start late read a
    normaliser that another block of the same run has already moved on, and nothing can be compared with them.)"""
    most = max(_cost(c) for c in listed())

    def log_int(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))
    while True:
        model = rng.choice(sorted(MODELS))
        cfg = MODELS[model]()
        room = min(4096, cfg.get("max_position_embeddings", 8192) - 40)
        case = {"model": model, "dtype": "bfloat16", "batch": log_int(1, 3 if model == "safuvik" else 64), "longest": log_int(1, room),
                "steps": rng.choice([0, rng.randint(1, 32)])}
        case["shortest"] = case["longest"] if rng.random() < 0.5 else log_int(1, case["longest"])
        if model.startswith("llama_tiny") or rng.random() < 0.15:
            case["dtype"] = "float32"
        logits = case["batch"] * (case["steps"] + 1) * (cfg.get("vocab") or cfg["vocab_size"]) * 4
        if _cost(case) <= most and logits <= 150e6 and sum(_lengths(case)) <= 17000:
            return case


# ------------------------------------------------------------------------------------------- inputs
def _lengths(case):
    r = random.Random("%d %d %d" % (case["batch"], case["shortest"], case["longest"]))
    return [case["longest"]] + [r.randint(case["shortest"], case["longest"]) for _ in range(case["batch"] - 1)]


def _spec(case):
    config = config_from_dict(MODELS[case["model"]]())
    return config, get_architecture(config.architecture).build_spec(config)


def _weights(case, seed):
    """Seeded weights on the GPU: matrices N(0, 0.02), norms 1 + N(0, 0.02), decays as trained models have them (memories of
    tens to thousands of tokens), and token embeddings that lean towards four experts' router rows each: a trained router
    is sure of its choice, and which experts run does not hang on the last bit."""
    _, spec = _spec(case)
    dtype = getattr(torch, case["dtype"])
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    def uniform(shape, lo, hi):
        return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo
    llama = "llama" in case["model"]
    out = {}
    for name, (shape, kind) in spec.tensor_table().items():
        shape = tuple(int(s) for s in shape)
        t = torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, 0.02, generator=g)
        if kind == "norm":
            t = t + 1
        elif kind in ("share", "taps"):
            t = t + 1.0 / shape[-1]
        elif kind == "identity":
            t = t + torch.eye(shape[-1], dtype=dtype, device="cuda")
        if name.endswith(".right.lam"):
            t = uniform(shape, -8.0, -3.5)
        elif name.endswith(".f.b"):
            t = uniform(shape, 3.0, 6.0)
        elif name.endswith(".A_log"):
            t = uniform(shape, 1.0, 16.0).log()
        elif name.endswith(".dt_bias"):
            t = torch.exp(uniform(shape, math.log(1e-3), math.log(1e-1))).expm1().log()
        elif name.endswith(".vmix"):
            t = uniform(shape, 0.3, 0.7)
        out[name] = t.to(dtype)
    routers = [n for n in out if n.endswith(".router")]
    if not llama:
        E = spec.width
        x = normal(spec.vocab_size, E)
        if routers:
            base = normal(*out[routers[0]].shape) * 0.02
            for n in routers:
                out[n] = (base + 0.1 * out[n].float()).to(dtype)
            R = torch.nn.functional.normalize(base, dim=1)
            picks = torch.rand(spec.vocab_size, R.shape[0], generator=g, device="cuda").topk(4, dim=1).indices
            x = x + 0.3 * math.sqrt(E) * R[picks].sum(1)
        out["embed"] = (x * (0.02 if spec.head_name is None else 1.0)).to(dtype)
    return out


def _tokens(case, seed):
    """Per sequence the prompt's ids and the ids that it is continued with."""
    _, spec = _spec(case)
    r = torch.Generator()
    r.manual_seed(seed ^ 0x5EED)
    return [(torch.randint(0, spec.vocab_size, (n,), generator=r).tolist(),
             torch.randint(0, spec.vocab_size, (case["steps"],), generator=r).tolist()) for n in _lengths(case)]


def prepare(case, seed):
    config, _ = _spec(case)
    pages = sum(-(-(n + case["steps"]) // 64) for n in _lengths(case))
    engine = Engine(config, _weights(case, seed), dtype=case["dtype"], max_tokens=64 * pages, max_batch=case["batch"])
    requests = _tokens(case, seed)
    if case["steps"]:                        # a server captures its decode step before the first request
        slots = [engine.new_sequence() for _ in requests]
        engine.step([StepEntry(s, p[:1], []) for s, (p, _) in zip(slots, requests)])
        engine.step([StepEntry(s, [c[0]], [0]) for s, (_, c) in zip(slots, requests)], captured=True)
        for s in slots:
            engine.end_sequence(s)
    return {"engine": engine, "requests": requests}


def run(state):
    """A batch of requests from prompts to the last step; logits [batch, vocab] after the prompts and after every step."""
    engine, requests = state["engine"], state["requests"]
    slots = [engine.new_sequence() for _ in requests]
    out = [engine.step([StepEntry(s, p, [len(p) - 1]) for s, (p, _) in zip(slots, requests)])]
    for k in range(len(requests[0][1])):
        out.append(engine.step([StepEntry(s, [c[k]], [0]) for s, (_, c) in zip(slots, requests)], captured=True))
    for s in slots:
        engine.end_sequence(s)
    return out


# ------------------------------------------------------------------------------------------- what a pass cannot do without
def _attentions(cfg):
    """(heads, values a score and a weighted sum cost together, values cached per position, window) per attention run."""
    if "num_hidden_layers" in cfg:
        d = cfg["head_dim"]
        return [(cfg["num_attention_heads"], 2 * d, 2 * cfg["num_key_value_heads"] * d, 0)] * cfg["num_hidden_layers"]
    loop = cfg.get("loop")
    order = list(range(len(cfg["layers"])))
    if loop:
        order = order[:loop["start"]] + order[loop["start"]:loop["stop"]] * loop["times"] + order[loop["stop"]:]
    out = []
    for i in order:
        m = cfg["layers"][i]["mixer"]
        m = m.get("left", m)
        if "scale" not in m:                 # a recurrence: its state does not grow with the position
            continue
        cached = m["kv_rank"] + m.get("rot_dim", 0) if "kv_rank" in m else m["kv_heads"] * (m["dim"] + m["vdim"])
        out.append((m["heads"], m["dim"] + m.get("rot_dim", 0) + m["vdim"], cached, (m.get("mask") or {}).get("size") or 0))
    return out


def work(case):
    """Every step reads every matrix that it multiplies by (of the experts those that some token can have chosen) and the
    cached positions; every token is multiplied by each matrix, wanted rows by the head."""
    cfg = MODELS[case["model"]]()
    _, spec = _spec(case)
    size = 4 if case["dtype"] == "float32" else 2
    lengths, steps = _lengths(case), case["steps"]
    table = spec.tensor_table()
    dense = routed = share = experts = 0
    for entry in spec.schedule:
        for name in set(spec.layers[entry.layer].names.values()):
            shape, _ = table[name]
            n = math.prod(shape) if len(shape) > 1 else 0
            if re.search(r"\.e\d+\.", name):
                routed += n
                r = next(la["mlp"]["router"] for la in cfg["layers"] if (la.get("mlp") or {}).get("kind") == "moe")
                share, experts = r["top"] / r["experts"], r["experts"]
            else:
                dense += n
    head = spec.vocab_size * spec.width
    tokens, batch = sum(lengths), case["batch"]
    flops = 2.0 * (dense + routed * share) * (tokens + steps * batch) + 2.0 * head * batch * (1 + steps)

    def touched(rows):
        return routed * (1.0 - (1.0 - share) ** rows) if experts else 0.0
    read = dense + touched(tokens) + head + steps * (dense + touched(batch) + head)
    moved = read * size + 4.0 * batch * (1 + steps) * spec.vocab_size
    for heads, both, cached, window in _attentions(cfg):
        for n in lengths:
            w = window or n + steps
            pairs = n * (n + 1) / 2 if n <= w else w * (w + 1) / 2 + (n - w) * w
            later = sum(min(w, n + k + 1) for k in range(steps))
            flops += 2.0 * heads * both * (pairs + later)
            moved += size * cached * (n + later + steps)
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["dtype"] == "float32":
        # measured against 64 bits: 3e-7 (the toy) to 9e-6 (4 layers of the 7B shape)
        return {"rel": 2e-5}
    # bf16 weights, activations, keys and values over 4 to 6 layers; measured against 64 bits: 0.009 to 0.018 for the Llama
    # shapes, whose layers' outputs outweigh the embedding, 0.002 to 0.009 for the others
    return {"rel": 0.025 if "llama" in case["model"] else 0.015, "max": 0.2}


# ------------------------------------------------------------------------------------------- the decoders in 64 bits
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(z):
    return z * torch.sigmoid(z)


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _softplus(z):
    return torch.nn.functional.softplus(z, threshold=50)


def _frequencies(rot):
    n, base = rot["dims"], rot["base"]
    f = base ** (-2.0 * torch.arange(n // 2, dtype=torch.float64, device="cuda") / n)
    sc = rot.get("scaling")
    if not sc:
        return f, 1.0
    if "low" in sc:                          # slow frequencies divided, a ramp between
        s = ((sc["original"] * f / (2.0 * math.pi) - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)
        return (1.0 - s) * f / sc["factor"] + s * f, 1.0

    def dim_of(turns):
        return n * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(dim_of(sc["fast"])), 0), min(math.ceil(dim_of(sc["slow"])), n - 1)
    r = ((torch.arange(n // 2, dtype=torch.float64, device="cuda") - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / sc["factor"] * r + f * (1.0 - r), 0.1 * math.log(sc["factor"]) + 1.0


def _turn(x, rot, interleaved=False):
    """x [T, heads, D]: the first rot["dims"] values of every head turned by the row's position."""
    n = rot["dims"]
    f, mag = _frequencies(rot)
    a = torch.arange(x.shape[0], dtype=torch.float64, device="cuda")[:, None] * f
    c, s = (torch.cos(a) * mag)[:, None], (torch.sin(a) * mag)[:, None]
    u, v = (x[..., 0:n:2], x[..., 1:n:2]) if interleaved else (x[..., :n // 2], x[..., n // 2:n])
    p, q = u * c - v * s, v * c + u * s
    both = torch.stack([p, q], dim=-1).flatten(-2) if interleaved else torch.cat([p, q], dim=-1)
    return torch.cat([both, x[..., n:]], dim=-1)


def _attend(q, k, v, scale, mask=None, softcap=None, sink=None):
    T, H = q.shape[:2]
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None]
    see = j <= i
    if mask and mask.get("size"):
        see = see & ((i - j < mask["size"]) | (j < (mask.get("keep_first") or 0)))
    out = torch.empty(T, H, v.shape[-1], dtype=q.dtype, device="cuda")
    for h in range(H):
        g = h // (H // k.shape[1])
        s = q[:, h] @ k[:, g].T * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], dim=1)
        out[:, h] = torch.softmax(s, dim=-1)[:, :T] @ v[:, g]
    return out


def _conv(x, taps):
    """Causal, per channel; the last tap is the row's own."""
    T, K = x.shape[0], taps.shape[1]
    padded = torch.cat([torch.zeros(K - 1, x.shape[1], dtype=x.dtype, device="cuda"), x])
    return sum(padded[j:j + T] * taps[:, j] for j in range(K))


def _decayed(q, k, v, decay):
    """S <- decay S + k v^T, o = S^T q; q, k [T, H, D], v [T, H, Dv], decay [T, H, D or 1]."""
    T, H, D = q.shape
    S = torch.zeros(H, D, v.shape[-1], dtype=q.dtype, device="cuda")
    out = torch.empty(T, H, v.shape[-1], dtype=q.dtype, device="cuda")
    for t in range(T):
        S = S * decay[t][:, :, None] + k[t][:, :, None] * v[t][:, None]
        out[t] = torch.bmm(q[t][:, None], S)[:, 0]
    return out


def _routed(h, ids, weights, expert, n):
    """Sum over the chosen of weight * expert(rows); ``ids`` >= n: the rows themselves."""
    out = torch.zeros_like(h)
    for e in range(int(ids.max()) + 1):
        rows, col = (ids == e).nonzero(as_tuple=True)
        if len(rows):
            y = expert(e, h[rows], weights[rows, col][:, None]) if e < n else weights[rows, col][:, None] * h[rows]
            out.index_add_(0, rows, y)
    return out


def _heads(x, n):
    return x.view(x.shape[0], n, -1)


def _safuvik_layer(layer, w, X, eps, cfg, shared):
    def mixer(h, m):
        T = h.shape[0]
        if layer["type"] == "mlstm":
            H, D, cap = m["heads"], m["dim"], m["gate_cap"]
            q, k, v = _heads(h @ w["mix.q"].T, H) * D ** -0.5, _heads(h @ w["mix.k"].T, H), _heads(h @ w["mix.v"].T, H)
            i = cap * torch.tanh((h @ w["mix.i"].T + w["mix.i.b"]) / cap)
            f = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w["mix.f"].T + w["mix.f.b"]) / cap))
            F = f.cumsum(0)                  # the running maximum of the exponents, from prefix sums
            top = torch.maximum(F + torch.cummax(i - F, 0).values, F)
            before = torch.cat([torch.zeros_like(top[:1]), top[:-1]])
            keep, take = torch.exp(f + before - top), torch.exp(i - top)
            one = torch.ones(T, H, 1, dtype=h.dtype, device="cuda")
            o = _decayed(q, k * take[..., None], torch.cat([v, one], -1), keep[..., None])
            o = o[..., :-1] / (torch.maximum(o[..., -1:].abs(), torch.exp(-top)[..., None]) + 1e-6)
            return (_rms(o, eps).reshape(T, -1) * w["mix.norm"] * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T
        p = m["left"]
        q, k = _rms(h @ w["mix.left.q"].T, eps) * w["mix.left.q.norm"], _rms(h @ w["mix.left.k"].T, eps) * w["mix.left.k.norm"]
        q, k = _turn(_heads(q, p["heads"]), p["rot"], True), _turn(_heads(k, p["kv_heads"]), p["rot"], True)
        o = _attend(q, k, _heads(h @ w["mix.left.v"].T, p["kv_heads"]), p["scale"], p["mask"])
        a = (o * torch.sigmoid(h @ w["mix.left.g"].T)[..., None]).reshape(T, -1) @ w["mix.left.o"].T
        B = m["right"]["blocks"]
        y = _gelu(h @ w["mix.right.y"].T + w["mix.right.y.b"])
        u = _conv(h @ w["mix.right.x"].T + w["mix.right.x.b"], w["mix.right.conv"]) + w["mix.right.conv.b"]

        def gate(n):
            return torch.sigmoid(torch.einsum("boi,tbi->tbo", w[n], _heads(u, B)) + w[n + ".b"]).reshape(T, -1)
        d = torch.exp(-8.0 * gate("mix.right.ra") * _softplus(w["mix.right.lam"]))
        drive = torch.sqrt(1.0 - d * d) * gate("mix.right.ri") * u
        S, states = torch.zeros_like(drive[0]), []
        for t in range(T):
            S = d[t] * S + drive[t]
            states.append(S)
        b = (torch.stack(states) * y) @ w["mix.right.o"].T
        return 0.5 * (_rms(a, eps) * w["mix.left.out"] + _rms(b, eps) * w["mix.right.out"])

    def ff(h, m):
        g, u = (h @ w["mlp.gate"].T).clamp(max=m["limit"]), (h @ w["mlp.up"].T).clamp(-m["limit"], m["limit"])
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w["mlp.down"].T
    if X.dim() == 2:
        X = X[None].repeat(cfg["streams"], 1, 1)
    for n, fn, m in (("1", mixer, layer["mixer"]), ("2", ff, layer["mlp"])):
        u = torch.einsum("s,ste->te", w[f"hc{n}.in"], X)
        y = fn(_rms(u, eps) * w["norm" + n], m)
        X = torch.einsum("st,sne->tne", w[f"hc{n}.mix"], X) + w[f"hc{n}.out"][:, None, None] * y
    return X


def _vaderax_layer(layer, w, x, eps, cfg, shared):
    def norm(x, n):
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w["norm" + n], w[f"norm{n}.b"], eps)
    h, m = norm(x, "1"), layer["mixer"]
    T, H, G = h.shape[0], m["heads"], m["kv_heads"]
    if layer["type"] == "attention":
        q, k = (_rms(_turn(_heads(h @ w["mix." + n].T, c), m["rot"]), eps) for n, c in (("q", H), ("k", G)))
        o = _attend(q, k, _heads(h @ w["mix.v"].T, G), m["scale"])
        y = (o.reshape(T, -1) * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T
    else:
        q, k, v = (_heads(_silu(_conv(h @ w["mix." + n].T, w[f"mix.{n}.conv"])), c) for n, c in (("q", G), ("k", G), ("v", H)))
        q, k = (z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6) for z in (q, k))
        q, k = (z.repeat_interleave(H // G, dim=1) for z in (q * m["dim"] ** -0.5, k))
        beta = torch.sigmoid(h @ w["mix.b"].T)
        g = torch.exp(-torch.exp(w["mix.A_log"]) * _softplus(h @ w["mix.a"].T + w["mix.dt_bias"]))
        S = torch.zeros(H, m["dim"], m["vdim"], dtype=h.dtype, device="cuda")
        o = torch.empty_like(v)
        for t in range(T):
            S = S * g[t][:, None, None]
            u = beta[t][:, None] * (v[t] - torch.bmm(k[t][:, None], S)[:, 0])
            S = S + k[t][:, :, None] * u[:, None]
            o[t] = torch.bmm(q[t][:, None], S)[:, 0]
        o = _rms(o, eps) * w["mix.norm"] * _silu(_heads(h @ w["mix.g"].T, H))
        y = o.reshape(T, -1) @ w["mix.o"].T
    x = x + y
    h, mlp = norm(x, "2"), layer["mlp"]
    if mlp["kind"] == "dense":
        return x + (h @ w["mlp.up"].T).clamp(min=0) ** 2 @ w["mlp.down"].T
    r = mlp["router"]
    s = torch.softmax(h @ w["mlp.router"].T, dim=-1)
    choice = (s + w["mlp.correction"]).view(T, r["groups"]["count"], -1)
    kept = choice.max(-1).values.topk(r["groups"]["keep"], dim=-1).indices
    bar = torch.full(choice.shape[:2], -math.inf, dtype=h.dtype, device="cuda").scatter_(1, kept, 0.0)
    ids = (choice + bar[..., None]).view(T, -1).topk(r["top"], dim=-1).indices
    return x + _routed(h, ids, s.gather(1, ids), lambda e, z, p: p * ((z @ w[f"mlp.e{e}.up"].T).clamp(min=0) ** 2
                                                                     @ w[f"mlp.e{e}.down"].T), r["experts"])


def _nifarax_layer(layer, w, x, eps, cfg, shared):
    def norm(x, n):
        return _rms(_heads(x, cfg["norm"]["groups"]), eps).reshape(x.shape) * w["norm" + n]

    def expert(z, pre, limit):
        g, u = (z @ w[pre + ".gate"].T).clamp(max=limit), (z @ w[pre + ".up"].T).clamp(-limit, limit)
        return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ w[pre + ".down"].T
    h, m = norm(x, "1"), layer["mixer"]
    T, H, gate = h.shape[0], m["heads"], torch.sigmoid(h @ w["rg1"].T + w["rg1.b"])
    h = h + _conv(h, w["canon1"])
    if layer["type"] == "gla":
        z = (h @ w["mix.a1"].T) @ w["mix.a2"].T + w["mix.a2.b"]
        o = _decayed(_heads(h @ w["mix.q"].T, H) * m["dim"] ** -0.5, _heads(h @ w["mix.k"].T, H), _heads(h @ w["mix.v"].T, H),
                     _heads(torch.sigmoid(z) ** (1.0 / m["tau"]), H))
        y = ((_rms(o, eps) * w["mix.norm"]).reshape(T, -1) * _silu(h @ w["mix.g"].T)) @ w["mix.o"].T
    else:
        q = _heads((_rms(h @ w["mix.dq"].T, eps) * w["mix.dq.norm"]) @ w["mix.uq"].T, H)
        c = _rms(h @ w["mix.dkv"].T, eps) * w["mix.dkv.norm"]
        o = _attend(q, _heads(c @ w["mix.uk"].T, H), _heads(c @ w["mix.uv"].T, H), m["scale"])
        y = o.reshape(T, -1) @ w["mix.o"].T
    x = x + y * gate
    h, mlp = norm(x, "2"), layer["mlp"]
    gate = torch.sigmoid(h @ w["rg2"].T + w["rg2.b"])
    h = h + _conv(h, w["canon2"])
    s, ids = torch.sigmoid(h @ w["mlp.router"].T).topk(mlp["router"]["top"], dim=-1)
    y = _routed(h, ids, s, lambda e, z, p: expert(p * z, f"mlp.e{e}", mlp["expert"]["limit"]), mlp["router"]["experts"])
    y = y + expert(h, "mlp.shared", mlp["shared"]["limit"]) * torch.sigmoid(h @ w["mlp.shared.sg"].T)
    return x + y * gate


def _gozotar_layer(layer, w, x, eps, cfg, shared):
    T, m = x.shape[0], layer["mixer"]
    if layer["type"] == "latent_attention":
        H, D, C = m["heads"], m["dim"], m["kv_rank"]
        q, down = _heads(x @ w["mix.q"].T, H), x @ w["mix.dkv"].T
        c = _rms(down[:, :C], eps) * w["mix.dkv.norm"]
        k_r = _turn(down[:, C:][:, None], m["rot"], True).expand(T, H, -1)
        q = torch.cat([q[..., :D], _turn(q[..., D:], m["rot"], True)], -1)
        o = _attend(q, torch.cat([_heads(c @ w["mix.uk"].T, H), k_r], -1), _heads(c @ w["mix.uv"].T, H), m["scale"],
                    sink=w["mix.sink"])
        y = o.reshape(T, -1) @ w["mix.o"].T
    elif layer["type"] == "attention":
        q, k = (_turn(_rms(_heads(x @ w["mix." + n].T, c), eps) * w[f"mix.{n}.norm"], m["rot"])
                for n, c in (("q", m["heads"]), ("k", m["kv_heads"])))
        v = _heads(x @ w["mix.v"].T, m["kv_heads"])
        if "first" in shared:
            v = (1.0 - w["mix.vmix"]) * v + w["mix.vmix"] * shared["first"]
        else:
            shared["first"] = v
        y = _attend(q, k, v, m["scale"], softcap=m["softcap"]).reshape(T, -1) @ w["mix.o"].T
    else:
        p, r = m["left"], m["right"]
        q, k = (_conv(x @ w["mix.left." + n].T, w[f"mix.left.{n}.conv"]) for n in "qk")
        v = _heads(k, p["kv_heads"])
        q, k = (_turn(_heads(_rms(z, eps) * w[f"mix.left.{n}.norm"], c), p["rot"])
                for z, n, c in ((q, "q", p["heads"]), (k, "k", p["kv_heads"])))
        o = _attend(q, k, v, p["scale"]) * torch.sigmoid(x @ w["mix.left.g"].T)[..., None]
        left = o.reshape(T, -1) @ w["mix.left.o"].T
        q, k = (_turn(_heads(x @ w["mix.right." + n].T, r["heads"]), r["rot"]) for n in "qk")
        decay = torch.tensor(r["decay"], dtype=x.dtype, device="cuda")[None, :, None].expand(T, -1, 1)
        o = _decayed(q, k * r["dim"] ** -0.5, _heads(x @ w["mix.right.v"].T, r["heads"]), decay)
        right = (_rms(o, eps).reshape(T, -1) * _silu(x @ w["mix.right.g"].T)) @ w["mix.right.o"].T
        y = m["left_scale"] * left + m["right_scale"] * right
    x = x + _rms(y, eps) * (1.0 + w["norm1"]) * w["ls1"]
    y = (_silu(x @ w["mlp.gate"].T) * (x @ w["mlp.up"].T)) @ w["mlp.down"].T
    x = x + _rms(y, eps) * (1.0 + w["norm2"]) * w["ls2"]
    y = (_gelu(x @ w["side.gate"].T) * shared["side"][shared["layer"]]) @ w["side.proj"].T
    return x + _rms(y, eps) * w["side.norm"]


def _busavik_layer(layer, w, x, eps, cfg, shared):
    def norm(x, n):
        return w["norm" + n] * torch.tanh(w[f"norm{n}.alpha"] * x) + w[f"norm{n}.b"]

    def expert(z, pre):
        return (_silu(z @ w[pre + ".gate"].T) * (z @ w[pre + ".up"].T)) @ w[pre + ".down"].T
    h, m, mlp = norm(x, "1"), layer["mixer"], layer["mlp"]
    T, H, D, C = h.shape[0], m["heads"], m["dim"], m["kv_rank"]
    q, down = _heads((_rms(h @ w["mix.dq"].T, eps) * w["mix.dq.norm"]) @ w["mix.uq"].T, H), h @ w["mix.dkv"].T
    c = _rms(down[:, :C], eps) * w["mix.dkv.norm"]
    k_r = _turn(down[:, C:][:, None], m["rot"]).expand(T, H, -1)
    q = torch.cat([q[..., :D], _turn(q[..., D:], m["rot"])], -1)
    o = _attend(q, torch.cat([_heads(c @ w["mix.uk"].T, H), k_r], -1), _heads(c @ w["mix.uv"].T, H), m["scale"])
    x = x + (o.reshape(T, -1) * torch.sigmoid(h @ w["mix.g"].T)) @ w["mix.o"].T
    h = norm(x, "2")
    if mlp["kind"] == "dense":
        y = _gelu(h @ w["mlp.gate"].T + w["mlp.gate.b"]) * (h @ w["mlp.up"].T + w["mlp.up.b"])
        return x + y @ w["mlp.down"].T + w["mlp.down.b"]
    z, ids = (h @ w["mlp.router"].T).topk(mlp["router"]["top"], dim=-1)
    y = _routed(h, ids, torch.softmax(z, -1), lambda e, z, p: p * expert(z, f"mlp.e{e}"), mlp["router"]["experts"])
    return x + y + torch.sigmoid(h @ w["mlp.shared.sg"].T) * expert(h, "mlp.shared")


def _bafulorn_layer(layer, w, x, eps, cfg, shared):
    def norm(x, n):
        return _rms(x, eps) * (1.0 + w["norm" + n])

    def expert(z, pre):
        return (_silu(z @ w[pre + ".gate"].T) * (z @ w[pre + ".up"].T)) @ w[pre + ".down"].T
    h, m, mlp = norm(x, "1"), layer["mixer"], layer["mlp"]
    T, H = h.shape[0], m["heads"]
    if layer["type"] == "latent_attention":
        c = _rms(h @ w["mix.dkv"].T, eps) * w["mix.dkv.norm"]
        o = _attend(_heads(h @ w["mix.q"].T, H), _heads(c @ w["mix.uk"].T, H), _heads(c @ w["mix.uv"].T, H), m["scale"], m["mask"])
        y = (o * torch.sigmoid(h @ w["mix.g"].T)[..., None]).reshape(T, -1) @ w["mix.o"].T
    elif layer["type"] == "attention":
        q, k = _heads(h @ w["mix.q"].T + w["mix.q.b"], H), _heads(h @ w["mix.k"].T + w["mix.k.b"], m["kv_heads"])
        o = _attend(_turn(q, m["rot"]), _turn(k, m["rot"]), k, m["scale"], m["mask"])
        y = o.reshape(T, -1) @ w["mix.o"].T + w["mix.o.b"]
    else:
        P, N, G = m["vdim"], m["state"], m["groups"]
        z, xbc, dt = (h @ w["mix.in"].T).split([H * P, H * P + 2 * G * N, H], dim=1)
        v, B, C = _silu(_conv(xbc, w["mix.conv"]) + w["mix.conv.b"]).split([H * P, G * N, G * N], dim=1)
        v, dt = _heads(v, H), _softplus(dt + w["mix.dt_bias"])
        B, C = (_heads(u, G).repeat_interleave(H // G, dim=1) for u in (B, C))
        o = _decayed(C, B * dt[..., None], v, torch.exp(-torch.exp(w["mix.A_log"]) * dt)[..., None]) + w["mix.D"][:, None] * v
        o = _rms(_heads(o.reshape(T, -1) * _silu(z), m["norm_groups"]), eps).reshape(T, -1) * w["mix.norm"]
        y = o @ w["mix.o"].T
    x = x + cfg["residual_mult"] * norm(y, "1b")
    h = norm(x, "2")
    if mlp["kind"] == "dense":
        y = ((h @ w["mlp.gate"].T).clamp(min=0) * (h @ w["mlp.up"].T)) @ w["mlp.down"].T
    else:
        r, s = mlp["router"], torch.sigmoid(h @ w["mlp.router"].T)
        ids = (s + w["mlp.correction"]).topk(r["top"], dim=-1).indices
        p = s.gather(1, ids)
        y = _routed(h, ids, p / (p.sum(-1, keepdim=True) + 1e-20) * r["scale"], lambda e, z, p: p * expert(z, f"mlp.e{e}"),
                    r["experts"]) + expert(h, "mlp.shared")
    return x + cfg["residual_mult"] * norm(y, "2b")


def _llama_layer(layer, w, x, eps, cfg, shared):
    T, H, G, D = x.shape[0], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    rot = {"base": cfg["rope_theta"], "dims": D}
    h = _rms(x, eps) * w["input_layernorm.weight"]
    q, k, v = (_heads(h @ w[f"self_attn.{n}_proj.weight"].T, c) for n, c in (("q", H), ("k", G), ("v", G)))
    o = _attend(_turn(q, rot), _turn(k, rot), v, D ** -0.5)
    x = x + o.reshape(T, -1) @ w["self_attn.o_proj.weight"].T
    h = _rms(x, eps) * w["post_attention_layernorm.weight"]
    y = _silu(h @ w["mlp.gate_proj.weight"].T) * (h @ w["mlp.up_proj.weight"].T)
    return x + y @ w["mlp.down_proj.weight"].T


def exact(case, seed):
    cfg, tensors = MODELS[case["model"]](), _weights(case, seed)
    llama = "num_hidden_layers" in cfg
    eps = cfg["rms_norm_eps"] if llama else cfg["norm"]["eps"]

    def of(prefix):
        return {k[len(prefix):]: v.double() for k, v in tensors.items() if k.startswith(prefix)}
    table = tensors["model.embed_tokens.weight" if llama else "embed"]
    requests = [p + c for p, c in _tokens(case, seed)]
    xs, shared = [], []
    for ids in requests:
        at = torch.tensor(ids, device="cuda")
        x, sh = table[at].double(), {}
        if cfg.get("architecture") == "Gozotar":
            b = cfg["embedding"]["bigram"]
            pairs = (at[:-1] * b["mul_prev"] + at[1:] * b["mul_cur"]) % b["buckets"]
            x = x + tensors["bigram"][torch.cat([pairs.new_tensor([b["buckets"]]), pairs])].double()
            sh["side"] = tensors["side.embed"][at].double().split(cfg["token_side"]["dim"], dim=1)
        elif cfg.get("architecture") == "Nifarax":
            x = _rms(_heads(x, cfg["norm"]["groups"]), eps).reshape(x.shape) * tensors["embed.norm"].double()
        elif cfg.get("architecture") == "Bafulorn":
            x = _rms(x, eps) * (1.0 + tensors["embed.norm"].double())
        xs.append(x)
        shared.append(sh)
    first = list(xs)
    order = list(range(cfg["num_hidden_layers"] if llama else len(cfg["layers"])))
    again = []
    if not llama and cfg.get("loop"):
        a, b, n = cfg["loop"]["start"], cfg["loop"]["stop"], cfg["loop"]["times"]
        order = order[:a] + order[a:b] * n + order[b:]
        again = [a + (b - a) * j for j in range(1, n)] if cfg["architecture"] == "Vaderax" else []
    one = {"Safuvik": _safuvik_layer, "Vaderax": _vaderax_layer, "Nifarax": _nifarax_layer, "Gozotar": _gozotar_layer,
           "Busavik": _busavik_layer, "Bafulorn": _bafulorn_layer}.get(cfg.get("architecture"), _llama_layer)
    for at, i in enumerate(order):
        layer = {} if llama else cfg["layers"][i]
        w = of("model.layers.%d." % i if llama else "l%d." % layer.get("weights_of", i))
        for n in range(len(xs)):
            shared[n]["layer"] = i
            xs[n] = one(layer, w, xs[n] + first[n] if at in again else xs[n], eps, cfg, shared[n])
    want = range(case["steps"] + 1)
    if "streams" in cfg:
        xs = [x.sum(0) for x in xs]
    x = torch.stack([x[len(ids) - case["steps"] - 1:] for x, ids in zip(xs, requests)])      # [batch, steps + 1, width]
    final = of("model.norm." if llama else "final.")
    if llama:
        x = _rms(x, eps) * final["weight"]
    elif cfg["architecture"] == "Vaderax":
        x = torch.nn.functional.layer_norm(x, x.shape[-1:], final["norm"], final["norm.b"], eps)
    elif cfg["architecture"] == "Busavik":
        x = final["norm"] * torch.tanh(final["norm.alpha"] * x) + final["norm.b"]
    elif cfg["architecture"] == "Nifarax":
        x = _rms(x.unflatten(-1, (cfg["norm"]["groups"], -1)), eps).flatten(-2) * final["norm"]
    else:
        x = _rms(x, eps) * (final["norm"] + (1.0 if cfg["architecture"] in ("Gozotar", "Bafulorn") else 0.0))
    head = table if not llama and cfg["architecture"] == "Nifarax" else tensors["lm_head.weight" if llama else "head"]
    head = head.double().T
    out = [x[:, k] @ head for k in want]
    if cfg.get("logit_softcap"):
        out = [cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"]) for z in out]
    return out
