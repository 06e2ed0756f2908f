"""What the speed of this library is measured on: calls of ``Engine.open``, ``Engine.step`` and ``Engine.close``.

A case is a model (a design of the library, its width, how many of its layers, its vocabulary, a dtype), a batch of
sequences and what is done with them: their prompts in one step, then ``new`` steps of one given token for every sequence,
then the sequences are closed.  That is what a program that scores, replays or generates does; with the tokens given, the
logits of every step can be compared.  The slots are opened and closed in every pass, so a pass leaves nothing behind.

The designs' sizes are those of the library's benchmark at widths 1,024 and 2,048.  Most cases run one layer of every kind that a
design has (three layers) with a small vocabulary, so that a layer's time and its rounding are what is seen; the whole
16-layer model of the benchmark stands for generation.  Weights are random with a standard deviation of 1 / sqrt(columns), so
that every part moves the stream by as much as it holds.  Prompts of a batch are of unequal lengths, in equal ratios from
``shortest`` to ``longest``.
"""
import math
from fractions import Fraction

import numpy as np
import torch
import torch.nn.functional as F

from mivi_v4_b200 import Engine
from mivi_v4_b200.engine.model import Model, describe_config, expected_tensors

DEVICE = "cuda:0"


def _case(name, design, width, layers, vocab, batch, shortest, longest, new, dtype="bfloat16", want="all"):
    return {"name": name, "design": design, "width": width, "layers": layers, "vocab": vocab, "dtype": dtype, "batch": batch,
            "shortest": shortest, "longest": longest, "new": new, "want": want}


def listed():
    return [
        # one user's reply from the whole 1.2B-parameter model: latency, launches, the weights' bytes
        _case("lfm2_reply_1", "lfm2", 2048, 16, 65536, 1, 29, 29, 16, want="last"),
        # the benchmark's batch: eight sequences decoded side by side
        _case("lfm2_replies_8", "lfm2", 2048, 16, 65536, 8, 48, 200, 16, want="last"),
        # a busy server: 64 unequal sequences, prompts in one step, then a few steps of 64 tokens
        _case("lfm2_replies_64", "lfm2", 2048, 16, 65536, 64, 7, 120, 16, want="last"),
        # prompts of unequal lengths scored in one step (the 700M-parameter layer sizes)
        _case("lfm2_score_unequal", "lfm2", 1536, 3, 2048, 12, 64, 2048, 0),
        # the 32-bit path (the 350M-parameter layer sizes): prompts of odd lengths, then a few tokens
        _case("lfm2_float32", "lfm2", 1024, 3, 2048, 4, 51, 700, 2, dtype="float32"),
        # a 2,048-token prompt through one layer of every kind of a design: linear recurrences and windowed attention ...
        _case("votavik_prompt", "votavik", 2048, 3, 2048, 1, 2048, 2048, 0),
        # ... state space, chunked attention beside a matrix memory, routed experts, prompts of two lengths
        _case("tevirax_prompts", "tevirax", 2048, 3, 2048, 2, 611, 1437, 0),
        # ... the delta rule with a decay a channel and latent attention with a window
        _case("puzorax_prompt", "puzorax", 2048, 3, 2048, 1, 2048, 2048, 0),
        # ... mixed heads beside a gated recurrence, distance-biased attention and the delta rule, at width 1,024, unequal prompts
        _case("ropelix_prompts", "ropelix", 1024, 3, 2048, 4, 130, 1500, 0),
        # ... latent attention of every earlier key and routed experts, a long prompt
        _case("redisun_long", "redisun", 2048, 3, 2048, 1, 6000, 6000, 0),
        # ... latent attention beside attention with a bias by distance, unequal prompts
        _case("mevulix_prompts", "mevulix", 2048, 3, 2048, 3, 333, 2048, 0),
        # short prompts and a few decoded tokens of a design with latent attention and experts
        _case("mevulix_replies_32", "mevulix", 2048, 3, 2048, 32, 9, 64, 8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Any design, either width, one layer of every kind; prompts of 33 to 6,000 tokens in all, or decoding of 1 to 64
    sequences, or (one in eight) the 32-bit path."""
    design = rng.choice(("lfm2", "votavik", "tevirax", "puzorax", "ropelix", "redisun", "mevulix"))
    width, vocab = rng.choice((1024, 2048)), rng.choice((1000, 2048, 4096))
    kind = rng.choice(("prompt",) * 4 + ("reply",) * 3 + ("float32",))
    if kind == "float32":
        n = _log_int(rng, 17, 600)
        return _bare("lfm2", width, vocab, rng.randint(1, 3), n, rng.randint(0, 2), "float32")
    if kind == "reply":
        batch = _log_int(rng, 1, 64)
        return _bare(design, width, vocab, batch, _log_int(rng, 16 * batch, 100 * batch), rng.randint(4, 12))
    return _bare(design, width, vocab, rng.choice((1, 1, 2, 3, 5)), _log_int(rng, 33, 3500), 0)


def _bare(design, width, vocab, batch, total, new, dtype="bfloat16"):
    mean = max(3, total // batch)
    c = _case("", design, width, 3, vocab, batch, max(2, int(mean * 0.4)) if batch > 1 else mean,
              int(mean * 1.7) if batch > 1 else mean, new, dtype)
    del c["name"]
    return c


# ---- the models ------------------------------------------------------------------------------------------------------
def _config(case):
    W, n, vocab = case["width"], case["layers"], case["vocab"]
    heads, kv, ff = W // 64, 8, 4 * W
    rot = {"dims": 32, "base": 1000000.0}
    moe = {"kind": "moe", "expert": {"ff": ff // 8}, "shared": {"ff": ff // 8}, "router": {"experts": 16, "top": 4}}
    d = case["design"]
    if d == "lfm2":
        pattern = ["conv", "conv", "full_attention", "conv", "conv", "full_attention", "conv", "conv", "full_attention", "conv",
                   "full_attention", "conv", "full_attention", "conv", "full_attention", "conv"]
        return {"architectures": ["Lfm2ForCausalLM"], "model_type": "lfm2", "hidden_size": W, "num_hidden_layers": n,
                "num_attention_heads": heads, "num_key_value_heads": kv, "vocab_size": vocab,
                "block_ff_dim": {1024: 6656, 1536: 10240, 2048: 12288}[W],
                "block_auto_adjust_ff_dim": True, "block_multiple_of": 256, "block_ffn_dim_multiplier": 1.0,
                "layer_types": pattern[:n], "rope_theta": 1000000.0, "norm_eps": 1e-5, "conv_L_cache": 3, "conv_bias": False,
                "tie_embedding": True}
    if d == "votavik":
        light = W // 128
        kinds = [
            {"type": "gla", "mlp": None, "mixer": {"heads": W // 256, "dim": 128, "vdim": 256, "tau": 8.0, "rank": 16}},
            {"type": "attention", "mlp": {"kind": "dense", "ff": ff, "limit": 7.0},
             "mixer": {"heads": heads, "kv_heads": kv, "dim": 80, "vdim": 64, "scale": 80 ** -0.5, "softcap": 30.0,
                       "mask": {"size": 1024, "keep_first": 64}, "rot": {"dims": 32, "base": 10000.0}}},
            {"type": "lightning", "mlp": None, "mixer": {"heads": light, "dim": 128, "vdim": 128,
                                                         "decay": [1.0 - 2.0 ** -(3 + 5 * i / light) for i in range(light)]}}]
        return {"architecture": "Votavik", "vocab": vocab, "width": W, "norm": {"eps": 1e-5}, "token_side": {"dim": 64},
                "layers": [kinds[i % 3] for i in range(n)]}
    if d == "tevirax":
        mamba = {"heads": 2 * W // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}
        par = {"left": {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 1024},
                        "rot": dict(rot, scaling={"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0})},
               "right": {"heads": W // 256, "dim": 128, "vdim": 256, "gate_cap": 15.0}, "left_scale": 1.0, "right_scale": 1.0}
        moe["router"]["groups"] = {"count": 4, "keep": 2}
        return {"architecture": "Tevirax", "vocab": vocab, "width": W, "max_positions": 8192, "norm": {"eps": 1e-6},
                "embedding": {"scale": float(W) ** 0.5}, "logit_softcap": 50.0,
                "layers": [{"type": "parallel" if i % 3 == 2 else "mamba2", "mixer": par if i % 3 == 2 else mamba,
                            "mlp": {"kind": "dense", "ff": ff} if i == 0 else moe} for i in range(n)]}
    if d == "puzorax":
        delta = {"heads": W // 128, "kv_heads": W // 256, "dim": 128, "vdim": 128, "conv": 4, "decay_rank": 64, "gate_rank": 64}
        latent = {"heads": heads, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 256, "scale": 96 ** -0.5,
                  "mask": {"size": 1024}, "rot": rot}
        moe = {"kind": "moe", "expert": {"ff": ff // 8}, "router": {"experts": 16, "identity": 2, "top": 4, "scale": 2.5}}
        return {"architecture": "Puzorax", "vocab": vocab, "width": W, "norm": {"eps": 1e-6},
                "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}},
                "layers": [{"type": "latent_attention" if i % 3 == 2 else "channel_delta", "mixer": latent if i % 3 == 2 else delta,
                            "mlp": moe} for i in range(n)]}
    if d == "ropelix":
        left = {"heads": heads, "kv_heads": kv // 4, "dim": 64, "vdim": 64, "scale": 0.125, "softcap": 30.0,
                "mask": {"size": 1024}, "rot": rot}
        par = {"left": left, "right": {"width": W, "blocks": W // 256, "conv": 4}, "left_scale": 1.0, "right_scale": 1.0}
        att = {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 64, "conv": 4, "scale": 0.125, "mask": {"size": 1024}}
        delta = {"heads": W // 128, "kv_heads": W // 256, "dim": 128, "vdim": 128, "conv": 4}
        kinds = (("parallel", par), ("attention", att), ("delta", delta))
        return {"architecture": "Ropelix", "vocab": vocab, "width": W, "norm": {"eps": 1e-6}, "embedding": {"scale": float(W) ** 0.5},
                "residual_mult": 0.5, "layers": [{"type": kinds[i % 3][0], "mixer": kinds[i % 3][1],
                                                  "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}} for i in range(n)]}
    latent = {"heads": heads, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 256, "q_rank": W // 4, "scale": 96 ** -0.5, "rot": rot}
    if d == "redisun":
        moe["expert"]["limit"] = moe["shared"]["limit"] = 7.0
        return {"architecture": "Redisun", "vocab": vocab, "width": W, "norm": {"eps": 1e-6}, "postln_alpha": 2.5,
                "embedding": {"bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}},
                "layers": [{"type": "latent_attention", "mixer": latent, "mlp": {"kind": "dense", "ff": ff} if i == 0 else moe}
                           for i in range(n)]}
    latent["rot"] = dict(rot, scaling={"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0})
    att = {"heads": heads, "kv_heads": kv, "dim": 64, "vdim": 64, "scale": 0.125, "softcap": 50.0,
           "q_temp": {"coef": 0.1, "every": 4096}, "bias_rows": 64, "bias_max": 256}
    return {"architecture": "Mevulix", "vocab": vocab, "width": W, "norm": {"eps": 1e-6}, "logit_scale": 0.5,
            "layers": [{"type": "attention" if i % 3 == 2 else "latent_attention", "mixer": att if i % 3 == 2 else latent,
                        "mlp": {"kind": "dense", "ff": ff} if i == 0 else moe} for i in range(n)]}


def _weights(case, seed):
    """Every tensor of the model, on the device, in the dtype it runs in."""
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    out = {}
    for name, spec in expected_tensors(_config(case)).items():
        mean, std = {"linear": (0.0, 0.0), "conv": (0.0, 0.0), "norm": (1.0, 0.1), "bias": (0.0, 0.1), "zeros": (0.0, 0.0)}[spec.init]
        if spec.init in ("linear", "conv"):
            std = spec.shape[-1] ** -0.5
        t = torch.randn(spec.shape, generator=gen, dtype=torch.float32, device=DEVICE) * std + mean
        out[name] = t.to(dtype) if spec.role == "matrix" else t
    return out


def _lengths(case):
    n, a, b = case["batch"], case["shortest"], case["longest"]
    return [a if n == 1 else int(round(a * (b / a) ** (i / (n - 1)))) for i in range(n)]


def _tokens(case, seed):
    """Every sequence's token ids: its prompt and the ``new`` tokens fed one a step."""
    rng = np.random.RandomState(seed % (1 << 32))
    return [rng.randint(0, case["vocab"], n + case["new"]) for n in _lengths(case)]


def prepare(case, seed):
    config, spec = describe_config(_config(case))
    model = Model(spec, config)
    model.load_params(_weights(case, seed), torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32, DEVICE)
    lens, tokens = _lengths(case), _tokens(case, seed)
    pages = sum(-(-len(t) // 64) for t in tokens)
    engine = Engine(model, max_tokens=64 * pages, max_batch=case["batch"])
    return {"engine": engine, "want": case["want"], "prompts": [t[:n] for t, n in zip(tokens, lens)],
            "steps": [[[int(t[n + s])] for t, n in zip(tokens, lens)] for s in range(case["new"])]}


def run(state):
    engine = state["engine"]
    slots = [engine.open() for _ in state["prompts"]]
    out = [engine.step(list(zip(slots, state["prompts"])), state["want"])]
    for tokens in state["steps"]:
        out.append(engine.step(list(zip(slots, tokens))))
    for s in slots:
        engine.close(s)
    return out


# ---- what a pass cannot do without -------------------------------------------------------------------------------------
def work(case):
    """Every weight read once a step (of an embedding table the step's rows only; of experts those that the step's tokens can
    reach), the logits and the cache's rows; two operations a weight and a token, and the mixers' own."""
    cfg, lens, new = _config(case), _lengths(case), case["new"]
    size = 2 if case["dtype"] == "bfloat16" else 4
    specs = expected_tensors(cfg)
    total = sum(lens)
    steps = [total] + [len(lens)] * new
    outs = [total if case["want"] == "all" else len(lens)] + [len(lens)] * new
    router = next((l["mlp"]["router"] for l in cfg["layers"] if (l.get("mlp") or {}).get("kind") == "moe"), None) if "layers" in cfg else None
    dense = routed = head = rows = 0
    for name, spec in specs.items():
        n = math.prod(spec.shape)
        if name in ("embed", "bigram", "pos", "side.embed", "model.embed_tokens.weight"):
            rows += spec.shape[-1]
            if name == "model.embed_tokens.weight" or (name == "embed" and "head" not in specs):
                head += n
        elif name == "head":
            head += n
        elif ".mlp.e" in name:
            routed += n
        elif spec.role == "matrix" or len(spec.shape) > 1:
            dense += n
    share = router["top"] / (router["experts"] + router.get("identity", 0)) if router else 0.0
    reached = [min(1.0, share * t) for t in steps]
    bytes_ = sum(size * (dense + routed * r + head + rows * t) for t, r in zip(steps, reached)) + sum(4 * case["vocab"] * o for o in outs)
    flops = sum(2 * t * (dense + routed * share) for t in steps) + sum(2 * o * head for o in outs)
    ends = [n + new for n in lens]
    for kind, m in _mixers(case, cfg):
        if kind == "full":
            H, dk, dv, row, window = m
            seen = sum(sum(min(p + 1, window) for p in range(e)) if window else e * (e + 1) // 2 for e in ends)
            flops += 2 * H * (dk + dv) * seen
            bytes_ += size * row * (total + sum(min(n + s + 1, window or n + s + 1) + 1 for n in lens for s in range(new)))
        else:
            H, dk, dv = m
            flops += 6 * H * dk * dv * sum(ends)
            bytes_ += 4 * H * dk * dv * len(lens) * (1 + 2 * new)
    return {"bytes": bytes_, "flops": flops}


def _mixers(case, cfg):
    """("full", (heads, key size, value size, cached numbers a token, window)) or ("state", (heads, key size, value size))."""
    if case["design"] == "lfm2":
        d = 64
        return [("full", (case["width"] // d, d, d, 2 * 8 * d, 0)) for k in cfg["layer_types"] if k == "full_attention"]
    out = []
    for l in cfg["layers"]:
        m = l["mixer"]
        for p in (m["left"], m["right"]) if l["type"] == "parallel" else (m,):
            if "kv_rank" in p:
                out.append(("full", (p["heads"], p["dim"] + p["rot_dim"], p["vdim"], p["kv_rank"] + p["rot_dim"], (p.get("mask") or {}).get("size", 0))))
            elif "scale" in p:
                out.append(("full", (p["heads"], p["dim"], p["vdim"], p["kv_heads"] * (p["dim"] + p["vdim"]), (p.get("mask") or {}).get("size", 0))))
            elif "state" in p:
                out.append(("state", (p["heads"], p["state"], p["vdim"])))
            elif "blocks" in p:
                out.append(("state", (p["width"], 1, 1)))
            else:
                out.append(("state", (p["heads"], p["dim"], p["vdim"])))
    return out


def tolerance(case):
    """Measured against ``exact``: 2.7e-6 in 32 bits; in bfloat16 0.0025 (ropelix), 0.006 (votavik), 0.007 (three lfm2 layers), 0.025
    (the whole model).  Where a router chooses experts, a token whose fourth and fifth experts nearly tie gets the other one
    under another rounding and its row is then off by about 0.3: 0.005 to 0.055 was seen over a whole output, and an output of
    few rows is off by that much as soon as it holds one such token."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    if case["design"] in ("tevirax", "puzorax", "redisun", "mevulix"):
        rows = case["batch"] if case["new"] or case["want"] == "last" else sum(_lengths(case))
        return {"rel": 0.1 + 0.3 / math.sqrt(rows)}
    return {"rel": {"ropelix": 0.01, "votavik": 0.025, "lfm2": 0.03 if case["layers"] <= 3 else 0.06}[case["design"]]}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------------
# x [B, T, width]: the sequences side by side, the shorter ones padded at their ends (no row sees a later one).
def exact(case, seed):
    lens, toks = _lengths(case), _tokens(case, seed)
    T = max(len(t) for t in toks)
    tokens = torch.zeros(len(toks), T, dtype=torch.long, device=DEVICE)
    for b, t in enumerate(toks):
        tokens[b, :len(t)] = torch.from_numpy(t).to(DEVICE)
    cfg = _config(case)
    w = {k: v.double() for k, v in _weights(case, seed).items()}
    f, head = _FORWARD[case["design"]](cfg, w, tokens)

    def logits(rows):
        return head(rows)
    first = torch.cat([f[b, :n] if case["want"] == "all" else f[b, n - 1:n] for b, n in enumerate(lens)])
    out = [logits(first)]
    for s in range(case["new"]):
        out.append(logits(torch.stack([f[b, n + s] for b, n in enumerate(lens)])))
    return out


def _sub(w, prefix):
    return {k[len(prefix):]: v for k, v in w.items() if k.startswith(prefix)}


def _lin(x, w):
    return x @ w.T


def _rms(x, eps, g=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if g is None else y * g


def _ln(x, g, b, eps):
    d = x - x.mean(-1, keepdim=True)
    y = d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * g
    return y if b is None else y + b


def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _turn(x, rot, neighbours=False):
    """x [B, T, heads, d]: the pairs (i, i + dims/2), or (2i, 2i + 1), of the first ``dims`` elements turn by the position."""
    if not rot:
        return x
    dims, sc = rot["dims"], rot.get("scaling")
    f = torch.tensor([rot["base"] ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=x.device)
    amp = 1.0
    if sc:
        def place(turns):
            return dims * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(rot["base"]))
        lo, hi = max(math.floor(place(sc["fast"])), 0), min(math.ceil(place(sc["slow"])), dims - 1)
        i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
        f, amp = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    a = (torch.arange(x.shape[1], dtype=torch.float64, device=x.device)[:, None] * f)[None, :, None, :]
    c, s = amp * torch.cos(a), amp * torch.sin(a)
    if neighbours:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        y = torch.stack([u * c - v * s, v * c + u * s], dim=-1).flatten(-2)
    else:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        y = torch.cat([u * c - v * s, v * c + u * s], dim=-1)
    return torch.cat([y, x[..., dims:]], dim=-1)


def _softmax(q, k, v, scale, window=0, keep=0, chunk=0, cap=0.0, sink=None, add=None, mix=None):
    """q [B, T, H, dk], k [B, T, G, dk], v [B, T, G, dv] -> [B, T, H * dv].  ``sink`` [H]: one more term exp(sink) in the
    denominator; ``add(h, distance)``: what is added to a head's scores; ``mix`` [H, H]: the heads' weights are mixed."""
    B, T, H, _ = q.shape
    G, dv = k.shape[2], v.shape[3]
    i, j = torch.arange(T, device=q.device)[:, None], torch.arange(T, device=q.device)[None, :]
    seen = j <= i
    if window:
        seen = seen & ((i - j < window) | (j < keep))
    if chunk:
        seen = seen & (i // chunk == j // chunk)
    dist = (i - j).clamp(min=0)
    out = torch.zeros(B, T, H, dv, dtype=q.dtype, device=q.device)
    for b in range(B):
        kept = []
        for h in range(H):
            g = h // (H // G)
            s = (q[b, :, h] @ k[b, :, g].T) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            if add is not None:
                s = s + add(h, dist)
            s = s.masked_fill(~seen, -math.inf)
            if sink is None:
                p = torch.softmax(s, dim=-1)
            else:
                top = torch.maximum(s.max(-1, keepdim=True).values, sink[h])
                e = torch.exp(s - top)
                p = e / (e.sum(-1, keepdim=True) + torch.exp(sink[h] - top))
            if mix is None:
                out[b, :, h] = p @ v[b, :, g]
            else:
                kept.append(p)
        if mix is not None:
            for g in range(G):                # sum over the heads of talk[h, a] (weights_a v_g)
                pv = torch.stack([p @ v[b, :, g] for p in kept])
                for h in range(g * (H // G), (g + 1) * (H // G)):
                    out[b, :, h] = torch.einsum("a,atd->td", mix[h], pv)
    return out.reshape(B, T, H * dv)


def _taps(x, taps, bias=None):
    K = taps.shape[-1]
    pad = F.pad(x, (0, 0, K - 1, 0))
    y = sum(pad[:, j:j + x.shape[1]] * taps[:, j] for j in range(K))
    return y if bias is None else y + bias


def _scan(q, k, v, a):
    """S <- a S + k v^T, o = S^T q; q, k [B, T, H, dk], v [B, T, H, dv], a [B, T, H, dk] or [B, T, H, 1]."""
    B, T, H, dk = k.shape
    S = torch.zeros(B, H, dk, v.shape[-1], dtype=q.dtype, device=q.device)
    out = torch.empty(B, T, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for t in range(T):
        S = a[:, t, :, :, None] * S + k[:, t, :, :, None] * v[:, t, :, None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
    return out


def _delta(q, k, v, beta, a):
    """S <- a S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q."""
    B, T, H, dk = k.shape
    S = torch.zeros(B, H, dk, v.shape[-1], dtype=q.dtype, device=q.device)
    out = torch.empty(B, T, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for t in range(T):
        S = S * a[:, t, :, :, None]
        u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ S)[:, :, 0])
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        out[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
    return out


def _glu(h, p, act, prefix=""):
    return _lin(act(_lin(h, p[prefix + "gate"]), _lin(h, p[prefix + "up"])), p[prefix + "down"])


def _silu_glu(g, u):
    return F.silu(g) * u


def _clamped(limit):
    def act(g, u):
        g = g.clamp(max=limit)
        return g * torch.sigmoid(1.702 * g) * (u.clamp(-limit, limit) + 1.0)
    return act


def _experts(h, weight, p, n, act, on_input=False):
    """The chosen experts of every token; weight [B, T, experts], zero where an expert is not chosen."""
    x, w = h.reshape(-1, h.shape[-1]), weight.reshape(-1, weight.shape[-1])
    y = torch.zeros_like(x)
    for e in range(n):
        at = torch.nonzero(w[:, e] != 0)[:, 0]
        if at.numel():
            we = w[at, e:e + 1]
            y[at] += _glu(x[at] * we, p, act, f"e{e}.") if on_input else we * _glu(x[at], p, act, f"e{e}.")
    return y.view_as(h)


def _heads(x, n):
    return x.view(*x.shape[:2], n, -1)


def _lfm2(cfg, w, tokens):
    eps, E = cfg["norm_eps"], w["model.embed_tokens.weight"]
    H, G = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    rot = {"dims": 64, "base": cfg["rope_theta"]}
    x = E[tokens]
    for i, kind in enumerate(cfg["layer_types"]):
        p = _sub(w, f"model.layers.{i}.")
        h = _rms(x, eps, p["operator_norm.weight"])
        if kind == "conv":
            b, c, u = _lin(h, p["conv.in_proj.weight"]).chunk(3, dim=-1)
            x = x + _lin(c * _taps(b * u, p["conv.conv.weight"][:, 0]), p["conv.out_proj.weight"])
        else:
            q = _turn(_rms(_heads(_lin(h, p["self_attn.q_proj.weight"]), H), eps, p["self_attn.q_layernorm.weight"]), rot, True)
            k = _turn(_rms(_heads(_lin(h, p["self_attn.k_proj.weight"]), G), eps, p["self_attn.k_layernorm.weight"]), rot, True)
            x = x + _lin(_softmax(q, k, _heads(_lin(h, p["self_attn.v_proj.weight"]), G), 0.125), p["self_attn.out_proj.weight"])
        h = _rms(x, eps, p["ffn_norm.weight"])
        x = x + _lin(F.silu(_lin(h, p["feed_forward.w1.weight"])) * _lin(h, p["feed_forward.w3.weight"]), p["feed_forward.w2.weight"])
    return _rms(x, eps, w["model.embedding_norm.weight"]), lambda r: _lin(r, E)


def _votavik(cfg, w, tokens):
    eps, x, side = cfg["norm"]["eps"], w["embed"][tokens], cfg["token_side"]["dim"]
    for i, c in enumerate(cfg["layers"]):
        t, m = _sub(w, f"l{i}."), c["mixer"]
        p, h = _sub(t, "mix."), _ln(x, t["norm1"], None, eps)
        H = m["heads"]
        if c["type"] == "gla":
            a = torch.sigmoid(_lin(_lin(h, p["a1"]), p["a2"]) + p["a2.b"]) ** (1.0 / m["tau"])
            o = _scan(_heads(_lin(h, p["q"]) * m["dim"] ** -0.5, H), _heads(_lin(h, p["k"]), H), _heads(_lin(h, p["v"]), H), _heads(a, H))
            y = (_rms(o, eps, p["norm"])).flatten(2) * F.silu(_lin(h, p["g"]))
        elif c["type"] == "lightning":
            q, k, v = (_heads(F.silu(_lin(h, p[n])), H) for n in "qkv")
            a = torch.tensor(m["decay"], dtype=x.dtype, device=x.device)[None, None, :, None].expand(*x.shape[:2], H, 1)
            y = _rms(_scan(q, k, v, a).flatten(2), eps, p["norm"]) * torch.sigmoid(_lin(h, p["g"]))
        else:
            G = m["kv_heads"]
            q = _turn(_heads(_rms(_lin(h, p["q"]), eps, p["q.norm"]), H), m["rot"])
            k = _turn(_heads(_rms(_lin(h, p["k"]), eps, p["k.norm"]), G), m["rot"])
            o = _softmax(q, k, _heads(_lin(h, p["v"]), G), m["scale"], m["mask"]["size"], m["mask"]["keep_first"], cap=m["softcap"], sink=p["sink"])
            y = (_heads(o, H) * torch.sigmoid(_lin(h, p["g"]))[..., None]).flatten(2)
        x = x + _lin(y, p["o"])
        if c["mlp"]:
            x = x + _glu(_ln(x, t["norm2"], None, eps), _sub(t, "mlp."), _clamped(c["mlp"]["limit"]))
        e = w["side.embed"][tokens][..., i * side:(i + 1) * side]
        x = x + _rms(_lin(_gelu(_lin(x, t["side.gate"])) * e, t["side.proj"]), eps, t["side.norm"])
    return _ln(x, w["final.norm"], None, eps), lambda r: _lin(r, w["head"])


def _tevirax(cfg, w, tokens):
    eps = cfg["norm"]["eps"]
    x = w["embed"][tokens] * cfg["embedding"]["scale"] + w["pos"][:tokens.shape[1]]
    for i, c in enumerate(cfg["layers"]):
        t, m = _sub(w, f"l{i}."), c["mixer"]
        p = _sub(t, "mix.")
        if c["type"] == "mamba2":
            H, inner, N = m["heads"], m["heads"] * m["vdim"], m["state"]
            z, xbc, dt = _lin(x, p["in"]).split([inner, inner + 2 * N, H], dim=-1)
            u, Bm, Cm = F.silu(_taps(xbc, p["conv"], p["conv.b"])).split([inner, N, N], dim=-1)
            u, dt = _heads(u, H), F.softplus(dt + p["dt_bias"], threshold=1e9)
            Bm, Cm = (n[:, :, None, :].expand(*n.shape[:2], H, N) for n in (Bm, Cm))
            o = _scan(Cm, Bm, u * dt[..., None], torch.exp(-torch.exp(p["A_log"]) * dt)[..., None]) + p["D"][:, None] * u
            y = _lin(_rms(o.flatten(2) * F.silu(z), eps, p["norm"]), p["o"])
        else:
            l, lp = m["left"], _sub(p, "left.")
            q = _turn(_rms(_heads(_lin(x, lp["q"]), l["heads"]), eps, lp["q.norm"]), l["rot"])
            k = _turn(_rms(_heads(_lin(x, lp["k"]), l["kv_heads"]), eps, lp["k.norm"]), l["rot"])
            left = _lin(_softmax(q, k, _heads(_lin(x, lp["v"]), l["kv_heads"]), l["scale"], chunk=l["mask"]["size"]), lp["o"])
            r, rp = m["right"], _sub(p, "right.")
            y = m["left_scale"] * left + m["right_scale"] * _lin(_memory(x, rp, r, eps), rp["o"])
        x = x + _rms(y, eps, t["norm1"])
        mlp, q = c["mlp"], _sub(t, "mlp.")
        if mlp["kind"] == "dense":
            y = _glu(x, q, _silu_glu)
        else:
            r = mlp["router"]
            s = torch.sigmoid(_lin(x, q["router"]))
            parts = s.view(*s.shape[:2], r["groups"]["count"], -1)
            best = parts.topk(2, dim=-1).values.sum(-1).topk(r["groups"]["keep"], dim=-1).indices
            allowed = torch.zeros(parts.shape[:3], dtype=torch.bool, device=x.device).scatter(2, best, True)
            pick = s.masked_fill(~allowed[..., None].expand_as(parts).reshape(s.shape), -math.inf).topk(r["top"], dim=-1).indices
            chosen = s.gather(-1, pick)
            weight = torch.zeros_like(s).scatter(-1, pick, chosen / (chosen.sum(-1, keepdim=True) + 1e-20))
            y = _experts(x, weight, q, r["experts"], _silu_glu) + torch.sigmoid(_lin(x, q["shared.sg"])) * _glu(x, q, _silu_glu, "shared.")
        x = x + _rms(y, eps, t["norm2"])
    cap = cfg["logit_softcap"]
    return _rms(x, eps, w["final.norm"]), lambda r: cap * torch.tanh(_lin(r, w["head"]) / cap)


def _memory(h, p, m, eps):
    """A matrix memory with exponential gates kept relative to a running maximum."""
    H, cap = m["heads"], m["gate_cap"]
    q, k, v = _heads(_lin(h, p["q"]) * m["dim"] ** -0.5, H), _heads(_lin(h, p["k"]), H), _heads(_lin(h, p["v"]), H)
    i = cap * torch.tanh((_lin(h, p["i"]) + p["i.b"]) / cap)
    f = F.logsigmoid(cap * torch.tanh((_lin(h, p["f"]) + p["f.b"]) / cap))
    B, T = h.shape[:2]
    S = torch.zeros(B, H, m["dim"], m["vdim"], dtype=h.dtype, device=h.device)
    n, top = torch.zeros(B, H, m["dim"], dtype=h.dtype, device=h.device), torch.zeros(B, H, dtype=h.dtype, device=h.device)
    out = torch.empty(B, T, H, m["vdim"], dtype=h.dtype, device=h.device)
    for t in range(T):
        new = torch.maximum(f[:, t] + top, i[:, t])
        a, b = torch.exp(f[:, t] + top - new)[..., None], torch.exp(i[:, t] - new)[..., None] * k[:, t]
        S, n, top = a[..., None] * S + b[..., None] * v[:, t, :, None, :], a * n + b, new
        den = torch.maximum((n * q[:, t]).sum(-1).abs(), torch.exp(-top)) + 1e-6
        out[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0] / den[..., None]
    return _rms(out, eps).flatten(2) * p["norm"] * torch.sigmoid(_lin(h, p["g"]))


def _bigram(cfg, w, tokens):
    bg = cfg["embedding"]["bigram"]
    rows = F.pad((tokens[:, :-1] * bg["mul_prev"] + tokens[:, 1:] * bg["mul_cur"]) % bg["buckets"], (1, 0), value=bg["buckets"])
    return w["embed"][tokens] + w["bigram"][rows]


def _latent(h, q, p, m, eps, neighbours=False, sink=None, window=0):
    H, dim = m["heads"], m["dim"]
    c, r = _lin(h, p["dkv"]).split([m["kv_rank"], m["rot_dim"]], dim=-1)
    c, r = _rms(c, eps, p["dkv.norm"]), _turn(r[:, :, None, :], m["rot"], neighbours)
    q = torch.cat([q[..., :dim], _turn(q[..., dim:], m["rot"], neighbours)], dim=-1)
    k = torch.cat([_heads(_lin(c, p["uk"]), H), r.expand(-1, -1, H, -1)], dim=-1)
    return _softmax(q, k, _heads(_lin(c, p["uv"]), H), m["scale"], window, sink=sink)


def _puzorax(cfg, w, tokens):
    eps, x = cfg["norm"]["eps"], _bigram(cfg, w, tokens)
    for i, c in enumerate(cfg["layers"]):
        t, m = _sub(w, f"l{i}."), c["mixer"]
        p, h, H = _sub(t, "mix."), _ln(x, t["norm1"], t["norm1.b"], eps), m["heads"]
        if c["type"] == "latent_attention":
            y = _latent(h, _heads(_lin(h, p["q"]), H), p, m, eps, sink=p["sink"], window=m["mask"]["size"]) * torch.sigmoid(_lin(h, p["g"]))
        else:
            a = _heads(_lin(_lin(h, p["a1"]), p["a2"]) + p["dt_bias"], H)
            g = torch.exp(-torch.exp(p["A_log"])[:, None] * F.softplus(a, threshold=1e9))
            o = _rms(_delta(*_delta_inputs(h, p, m), torch.sigmoid(_lin(h, p["b"])), g), eps, p["norm"])
            y = o.flatten(2) * torch.sigmoid(_lin(_lin(h, p["g1"]), p["g2"]))
        y = _lin(y, p["o"])
        q, r = _sub(t, "mlp."), c["mlp"]["router"]
        s = torch.softmax(_lin(h, q["router"]), dim=-1)
        pick = (s + q["correction"]).topk(r["top"], dim=-1).indices
        chosen = s.gather(-1, pick)
        weight = torch.zeros_like(s).scatter(-1, pick, chosen / (chosen.sum(-1, keepdim=True) + 1e-20) * r["scale"])
        x = x + y + _experts(h, weight, q, r["experts"], _silu_glu) + weight[..., r["experts"]:].sum(-1, keepdim=True) * h
    return _ln(x, w["final.norm"], w["final.norm.b"], eps), lambda r: _lin(r, w["head"])


def _delta_inputs(h, p, m):
    def unit(x):
        return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    H, G = m["heads"], m["kv_heads"]
    q, k = (unit(_heads(F.silu(_taps(_lin(h, p[n]), p[n + ".conv"])), G)).repeat_interleave(H // G, dim=2) for n in "qk")
    return q * m["dim"] ** -0.5, k, _heads(F.silu(_taps(_lin(h, p["v"]), p["v.conv"])), H)


def _ropelix(cfg, w, tokens):
    eps, mult, x = cfg["norm"]["eps"], cfg["residual_mult"], w["embed"][tokens] * cfg["embedding"]["scale"]
    for i, c in enumerate(cfg["layers"]):
        t, m = _sub(w, f"l{i}."), c["mixer"]
        p, h = _sub(t, "mix."), _rms(x, eps, 1.0 + t["norm1"])
        if c["type"] == "parallel":
            l, lp = m["left"], _sub(p, "left.")
            q = _turn(_heads(_rms(_lin(h, lp["q"]), eps, lp["q.norm"]), l["heads"]), l["rot"])
            k = _turn(_heads(_rms(_lin(h, lp["k"]), eps, lp["k.norm"]), l["kv_heads"]), l["rot"])
            o = _softmax(q, k, _heads(_lin(h, lp["v"]), l["kv_heads"]), l["scale"], l["mask"]["size"], cap=l["softcap"], mix=lp["talk"])
            rp = _sub(p, "right.")
            u = _taps(_lin(h, rp["x"]) + rp["x.b"], rp["conv"], rp["conv.b"])
            r, g = (torch.sigmoid((torch.einsum("btni,noi->btno", _heads(u, m["right"]["blocks"]), rp[n]) + rp[n + ".b"]).flatten(2)) for n in ("ra", "ri"))
            log_a = -8.0 * r * F.softplus(rp["lam"], threshold=1e9)
            a, b = torch.exp(log_a), torch.sqrt(-torch.expm1(2.0 * log_a)) * g * u
            S, states = torch.zeros_like(u[:, 0]), []
            for s in range(u.shape[1]):
                S = a[:, s] * S + b[:, s]
                states.append(S)
            right = _lin(torch.stack(states, dim=1) * _gelu(_lin(h, rp["y"]) + rp["y.b"]), rp["o"])
            y = m["left_scale"] * _lin(o, lp["o"]) + m["right_scale"] * right
        elif c["type"] == "attention":
            q = _heads(_taps(_lin(h, p["q"]), p["q.conv"]), m["heads"])
            k = _heads(_taps(_lin(h, p["k"]), p["k.conv"]), m["kv_heads"])
            o = _softmax(q, k, k[..., :m["vdim"]], m["scale"], m["mask"]["size"], sink=torch.zeros_like(p["r1"]),
                         add=lambda a, n: -p["r1"][a] * torch.log1p(p["r2"][a] * n))
            y = _lin(o * torch.sigmoid(_lin(h, p["g"])), p["o"])
        else:
            g = torch.exp(-torch.exp(p["A_log"]) * F.softplus(_lin(h, p["a"]) + p["dt_bias"], threshold=1e9))[..., None]
            o = _rms(_delta(*_delta_inputs(h, p, m), torch.sigmoid(_lin(h, p["b"])), g), eps, p["norm"])
            y = _lin(o.flatten(2) * F.silu(_lin(h, p["g"])), p["o"])
        x = x + mult * t["ls1"] * y
        x = x + mult * t["ls2"] * _glu(_rms(x, eps, 1.0 + t["norm2"]), _sub(t, "mlp."), _clamped(c["mlp"]["limit"]))
    return _rms(x, eps, 1.0 + w["final.norm"]), lambda r: _lin(r, w["embed"])


def _redisun(cfg, w, tokens):
    eps, alpha, x = cfg["norm"]["eps"], cfg["postln_alpha"], _bigram(cfg, w, tokens)
    for i, c in enumerate(cfg["layers"]):
        t, m = _sub(w, f"l{i}."), c["mixer"]
        p, H = _sub(t, "mix."), m["heads"]
        o = _latent(x, _heads(_lin(_rms(_lin(x, p["dq"]), eps, p["dq.norm"]), p["uq"]), H), p, m, eps, sink=p["sink"])
        y = _lin((_heads(o, H) * torch.sigmoid(_lin(x, p["g"]))[..., None]).flatten(2), p["o"])
        x = _rms(alpha * x + torch.sigmoid(_lin(x, t["rg1"]) + t["rg1.b"]) * y, eps, t["norm1"])
        q, mlp = _sub(t, "mlp."), c["mlp"]
        if mlp["kind"] == "dense":
            y = _glu(x, q, _silu_glu)
        else:
            best = (_lin(x, q["router"]) + q["router.b"]).topk(mlp["router"]["top"], dim=-1)
            weight = torch.zeros(*x.shape[:2], mlp["router"]["experts"], dtype=x.dtype, device=x.device)
            weight = weight.scatter(-1, best.indices, torch.softmax(best.values, dim=-1))
            act = _clamped(mlp["expert"]["limit"])
            y = _experts(x, weight, q, mlp["router"]["experts"], act) + _glu(x, q, act, "shared.")
        x = _rms(alpha * x + torch.sigmoid(_lin(x, t["rg2"]) + t["rg2.b"]) * y, eps, t["norm2"])
    return _rms(x, eps, w["final.norm"]), lambda r: _lin(r, w["head"])


def _bucket(n, rows, reach):
    """The row of the bias table for a key ``n`` tokens back: one each for the nearest, then ever longer stretches."""
    half = rows // 2
    if n < half:
        return n
    k, have, unit = 0, (Fraction(n) / half) ** (rows - half), Fraction(reach) / half
    while half + k + 1 <= rows - 1 and have >= unit ** (k + 1):
        k += 1
    return half + k


def _mevulix(cfg, w, tokens):
    eps, x = cfg["norm"]["eps"], w["embed"][tokens]
    for i, c in enumerate(cfg["layers"]):
        t, m = _sub(w, f"l{i}."), c["mixer"]
        p, H = _sub(t, "mix."), m["heads"]
        if c["type"] == "attention":
            pos = torch.arange(x.shape[1], device=x.device)
            temp = 1.0 + m["q_temp"]["coef"] * torch.log(((pos + 1) // m["q_temp"]["every"] + 1).double())
            q = _heads(_rms(_lin(x, p["q"]) + p["q.b"], eps, p["q.norm"]) * temp[:, None], H)
            k = _heads(_rms(_lin(x, p["k"]) + p["k.b"], eps, p["k.norm"]), m["kv_heads"])
            v = _heads(_lin(x, p["v"]) + p["v.b"], m["kv_heads"])
            rows = torch.tensor([_bucket(n, m["bias_rows"], m["bias_max"]) for n in range(m["bias_max"] + 1)], device=x.device)
            y = _softmax(q, k, v, m["scale"], cap=m["softcap"], sink=p["sink"],
                         add=lambda h, n: p["rel"][:, h][rows[n.clamp(max=m["bias_max"])]])
        else:
            y = _latent(x, _heads(_lin(_rms(_lin(x, p["dq"]), eps, p["dq.norm"]), p["uq"]), H), p, m, eps, neighbours=True)
        x = x + t["ls1"] * _ln(_lin(y, p["o"]), t["norm1"], t["norm1.b"], eps)
        q, mlp = _sub(t, "mlp."), c["mlp"]
        if mlp["kind"] == "dense":
            y = _glu(x, q, lambda g, u: _gelu(g) * u)
        else:
            z = _lin(x, q["router"])
            pick = z.topk(mlp["router"]["top"], dim=-1).indices
            weight = torch.zeros_like(z).scatter(-1, pick, torch.sigmoid(z.gather(-1, pick)))
            y = _experts(x, weight, q, mlp["router"]["experts"], _silu_glu, on_input=True) + _glu(x, q, _silu_glu, "shared.")
        x = x + t["ls2"] * _ln(y, t["norm2"], t["norm2.b"], eps)
    return _ln(x, w["final.norm"], w["final.norm.b"], eps), lambda r: _lin(r, w["head"]) * cfg["logit_scale"]


_FORWARD = {"lfm2": _lfm2, "votavik": _votavik, "tevirax": _tevirax, "puzorax": _puzorax, "ropelix": _ropelix, "redisun": _redisun,
            "mevulix": _mevulix}
