"""Workloads of this engine, for timing: what a program that serves or scores models with it has it do.

Two kinds of case.  `part` 'step' is a whole decode step of a Qwen3 model through `ModelRunner.prepare` and
`ModelRunner.forward`, host work and captured graphs included, and returns the logits beside the pages.  Every other part is one mixer or
feed-forward of a one-layer model, called as a model's layers call it (`forward(x, ctx)` for a batch that the step
function prepared, `forward(x)` for a feed-forward), and returns what joins the residual stream, beside the pages or
states that it wrote.  Sizes are those of bench.py: the Qwen3-0.6B and Qwen3-8B layer shapes, and the layers of the other
designs at widths 1,024, 2,048 and 4,096 with heads of 128.

Fields of a case: `part`, `dtype`, `width`, `tokens` (new tokens in the step), `requests` they belong to (the portions are
uneven), `context` (tokens each request has cached already, uneven too), and `layers` for whole steps.  A request with one
new token is decoding.  Weights have a standard deviation of 1 / sqrt(inputs), activations one of 1, as normed layers see.
"""
import math

import numpy as np
import torch

from litellmengine_b200.config import config_from_dict
from litellmengine_b200.engine import ModelRunner, StepEntry
from litellmengine_b200.weights import DictSource

DEVICE = "cuda"
F64 = torch.float64
HEAD = 128
PAGE = 16
SIZES = {1024: (3072, 8, 4), 2048: (6144, 16, 8), 4096: (12288, 32, 8)}     # feed-forward, query heads, kv heads
QWEN_HEADS = {1024: (16, 8), 4096: (32, 8)}                                   # the 0.6B and the 8B shape
STEP_VOCAB = {1024: 151936, 4096: 32768}     # the 0.6B shape's own tied head; a smaller one beside a cut of the 8B shape
THETA = 1000000.0
LATENT_RANK, LATENT_ROT = 512, 64
RANK, TAPS, TAU = 64, 4, 8.0                 # low-rank projections and convolutions of the recurrent mixers
WINDOW, KEEP_FIRST = 1024, 4
EXPERTS, TOP, LIMIT = 8, 2, 7.0
EPS = {"qwen": 1e-6, "design": 1e-5}
PORTION = 8192                               # most tokens of one step


def listed():
    c = lambda name, part, dtype, width, tokens, requests, context, layers=1: dict(
        name=name, part=part, dtype=dtype, width=width, tokens=tokens, requests=requests, context=context, layers=layers)
    return [
        # a small model's decode step of a few chats: latency and launches
        c("step_small", "step", "bfloat16", 1024, 5, 5, 320, 8),
        # the 32-bit mode (the number format of the engine this one replaces), decoding at the 8B layer sizes
        c("step_float32", "step", "float32", 4096, 8, 8, 1500, 4),
        # a prompt that continues a cached one, beside a shorter one
        c("attention_prompt", "attention", "bfloat16", 4096, 2900, 2, 700),
        # decoding of many chats at a long context: the cache is what is read
        c("attention_decode", "attention", "bfloat16", 4096, 45, 45, 3900),
        # a prompt in the 32-bit mode
        c("attention_prompt_float32", "attention", "float32", 4096, 500, 1, 0),
        # the dense feed-forward between the smallest decode steps and prompts, and in a prompt
        c("mlp_decode", "mlp", "bfloat16", 4096, 40, 40, 0),
        c("mlp_prompt", "mlp", "bfloat16", 4096, 2045, 1, 0),
        # attention over cached latents, a whole prompt
        c("latent_prompt", "latent", "bfloat16", 4096, 2000, 1, 0),
        # recurrent mixers over a prompt, and over the prompts of several requests
        c("gla_prompt", "gla", "bfloat16", 4096, 2048, 1, 0),
        c("delta_prompt", "delta", "bfloat16", 4096, 1700, 3, 0),
        # attention in a window that keeps the first keys, with learned sinks
        c("windowed_prompt", "windowed", "bfloat16", 4096, 2500, 1, 0),
        # routed experts when a few dozen requests decode
        c("experts_decode", "experts", "bfloat16", 2048, 24, 24, 0),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    part = rng.choice(("step", "step", "attention", "attention", "mlp", "mlp", "latent", "gla", "delta", "windowed", "experts"))
    dtype = rng.choice(("bfloat16", "bfloat16", "float32")) if part in ("step", "attention", "mlp") else "bfloat16"
    narrow = dtype == "float32"
    layers = 1
    if part == "step":
        width, layers = (4096, rng.randint(1, 4)) if narrow else (1024, rng.randint(4, 12))
        requests = log(1, 8 if narrow else 32)
        tokens, context = requests, log(16, 1500 if narrow else 512)
    else:
        width = 4096 if part in ("attention", "mlp") else rng.choice((1024, 2048, 4096))
        if part in ("mlp", "experts"):
            tokens = log(1, 512 if narrow else 2048)
            requests, context = 1, 0
        elif rng.random() < 0.5:                          # decoding
            requests = log(1, 8 if narrow else 64)
            tokens, context = requests, log(16, 1500 if narrow else 3900)
        else:                                             # prompts
            tokens = log(16, 500 if narrow else 3000 if part == "attention" else 2500)
            requests = min(tokens, rng.choice((1, 1, 2, 3)))
            context = 0 if narrow else rng.choice((0, 0, log(16, 1000)))
    return dict(part=part, dtype=dtype, width=width, tokens=tokens, requests=requests, context=context, layers=layers)


# ---- sizes ------------------------------------------------------------------------------------------------
def _portions(case):
    """New tokens of each request: 1 : 2 : 3 ... as near as whole numbers come, all of them at least 1."""
    n, total = case["requests"], case["tokens"]
    got = [1 + (total - n) * (i + 1) * 2 // (n * (n + 1)) for i in range(n)]
    got[-1] += total - sum(got)
    return got


def _contexts(case):
    """Cached tokens of each request: between three quarters of `context` and all of it."""
    c, n = case["context"], case["requests"]
    return [c - (c // 4) * i // n for i in range(n)]


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32


def _config(case):
    part, W = case["part"], case["width"]
    ff, heads, kv = SIZES[W]
    if part in ("step", "attention", "mlp"):
        heads, kv = QWEN_HEADS[W]
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=case["layers"], hidden_size=W,
                    num_attention_heads=heads, num_key_value_heads=kv, head_dim=HEAD, intermediate_size=ff,
                    vocab_size=STEP_VOCAB[W] if part == "step" else 64, rope_theta=THETA, rms_norm_eps=EPS["qwen"],
                    max_position_embeddings=40960, tie_word_embeddings=part == "step" and W == 1024, torch_dtype=case["dtype"])
    half, mlp = max(1, heads // 2), None
    rot = {"base": 10000.0, "dims": LATENT_ROT}
    if part == "latent":
        name, kind, mixer = "Vugedra", "latent_attention", {
            "heads": heads, "dim": HEAD, "rot_dim": LATENT_ROT, "vdim": HEAD, "q_rank": 3 * W // 8, "kv_rank": LATENT_RANK,
            "scale": (HEAD + LATENT_ROT) ** -0.5, "rot": rot}
    elif part == "gla":
        name, kind, mixer = "Vugedra", "gla", {"heads": half, "dim": HEAD, "vdim": HEAD, "tau": TAU, "rank": RANK}
    elif part == "delta":
        name, kind, mixer = "Pukatar", "channel_delta", {"heads": half, "kv_heads": half, "dim": HEAD, "vdim": HEAD, "conv": TAPS,
                                                         "decay_rank": RANK, "gate_rank": RANK}
    else:
        name, kind, mixer = "Pukatar", "attention", {"heads": heads, "kv_heads": kv, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5,
                                                     "mask": {"size": WINDOW, "keep_first": KEEP_FIRST}, "rot": rot}
    if part == "experts":
        mlp = {"kind": "moe", "expert": {"ff": ff // 2, "limit": LIMIT}, "router": {"experts": EXPERTS, "top": TOP},
               "shared": {"ff": ff // 4, "limit": LIMIT}}
    return {"architecture": name, "vocab": 64, "width": W, "norm": {"eps": EPS["design"]},
            "layers": [{"type": kind, "mixer": mixer, "mlp": mlp}]}


def _shapes(case):
    """name -> (shape, kind) of the tensors the timed part reads; kind 'matrix', 'one' (1 + 0.1 n) or a standard deviation."""
    part, W = case["part"], case["width"]
    ff, heads, kv = SIZES[W]
    half, out = max(1, heads // 2), {}
    if part in ("step", "attention", "mlp"):
        heads, kv = QWEN_HEADS[W]
        for i in range(case["layers"]):
            p = f"model.layers.{i}."
            for n, shape in (("q", (heads * HEAD, W)), ("k", (kv * HEAD, W)), ("v", (kv * HEAD, W)), ("o", (W, heads * HEAD))):
                out[f"{p}self_attn.{n}_proj.weight"] = (shape, "matrix")
            out[p + "self_attn.q_norm.weight"] = out[p + "self_attn.k_norm.weight"] = ((HEAD,), "one")
            for n, shape in (("gate", (ff, W)), ("up", (ff, W)), ("down", (W, ff))):
                out[f"{p}mlp.{n}_proj.weight"] = (shape, "matrix")
            out[p + "input_layernorm.weight"] = out[p + "post_attention_layernorm.weight"] = ((W,), "one")
        if part == "step":
            out["model.embed_tokens.weight"] = ((STEP_VOCAB[W], W), "matrix")
            out["model.norm.weight"] = ((W,), "one")
            if W != 1024:
                out["lm_head.weight"] = ((STEP_VOCAB[W], W), "matrix")
        return out
    p = "l0.mix."
    if part == "latent":
        Q, R, P = 3 * W // 8, LATENT_RANK, LATENT_ROT
        for n, shape in (("dq", (Q, W)), ("uq", (heads * (HEAD + P), Q)), ("dkv", (R + P, W)), ("uk", (heads * HEAD, R)),
                         ("uv", (heads * HEAD, R)), ("g", (heads, W)), ("o", (W, heads * HEAD))):
            out[p + n] = (shape, "matrix")
        out[p + "dq.norm"], out[p + "dkv.norm"] = ((Q,), "one"), ((R,), "one")
    elif part == "gla":
        hd = half * HEAD
        for n, shape in (("q", (hd, W)), ("k", (hd, W)), ("v", (hd, W)), ("g", (hd, W)), ("a1", (RANK, W)), ("o", (W, hd))):
            out[p + n] = (shape, "matrix")
        out[p + "a2"], out[p + "a2.b"], out[p + "norm"] = ((hd, RANK), RANK ** -0.5), ((hd,), 0.5), ((HEAD,), "one")
    elif part == "delta":
        hd = half * HEAD
        for n, shape in (("q", (hd, W)), ("k", (hd, W)), ("v", (hd, W)), ("b", (half, W)), ("a1", (RANK, W)), ("a2", (hd, RANK)),
                         ("g1", (RANK, W)), ("g2", (hd, RANK)), ("o", (W, hd))):
            out[p + n] = (shape, "matrix")
        for n in ("q.conv", "k.conv", "v.conv"):
            out[p + n] = ((hd, TAPS), 0.5)
        out[p + "dt_bias"], out[p + "A_log"], out[p + "norm"] = ((hd,), 1.0), ((half,), 0.5), ((HEAD,), "one")
    else:
        for n, shape in (("q", (heads * HEAD, W)), ("k", (kv * HEAD, W)), ("v", (kv * HEAD, W)), ("o", (W, heads * HEAD))):
            out[p + n] = (shape, "matrix")
        out[p + "sink"] = ((heads,), 1.0)
    if part == "experts":
        m, fe, fs = "l0.mlp.", ff // 2, ff // 4
        out[m + "router"], out[m + "router.b"], out[m + "shared.sg"] = ((EXPERTS, W), W ** -0.5), ((EXPERTS,), 0.1), ((1, W), W ** -0.5)
        for e, f in [(f"e{e}.", fe) for e in range(EXPERTS)] + [("shared.", fs)]:
            out[m + e + "gate"], out[m + e + "up"], out[m + e + "down"] = ((f, W), "matrix"), ((f, W), "matrix"), ((W, f), "matrix")
    return out


# ---- inputs -----------------------------------------------------------------------------------------------
def _generator(seed, stream):
    return torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + stream) % (1 << 62))


def _weights(case, seed):
    g, out = _generator(seed, 1), {}
    for name, (shape, kind) in _shapes(case).items():
        t = torch.randn(shape, generator=g, device=DEVICE)
        if kind == "one":
            t = t.mul_(0.1).add_(1.0)
        elif kind == "matrix":
            t = t.mul_(shape[1] ** -0.5).to(_dtype(case))
        else:
            t = t.mul_(kind)
        out[name] = t
    return out


def _rows(case, seed):
    """Per request the layer inputs of its whole sequence, cached tokens first (token ids for whole steps)."""
    g, out = _generator(seed, 2), []
    for past, new in zip(_contexts(case), _portions(case)):
        if case["part"] == "step":
            out.append(torch.randint(0, STEP_VOCAB[case["width"]], (past + new,), generator=g, device=DEVICE))
        else:
            out.append(torch.randn(past + new, case["width"], generator=g, device=DEVICE).to(_dtype(case)))
    return out


def prepare(case, seed):
    """The model with its cache, and requests whose earlier tokens are in it."""
    weights, rows = _weights(case, seed), _rows(case, seed)
    config = config_from_dict(_config(case))
    part, past, new = case["part"], _contexts(case), _portions(case)
    params = _rest(config, weights, _dtype(case))
    held = sum(-(-(p + n) // PAGE) * PAGE for p, n in zip(past, new))
    runner = ModelRunner.from_config(config, dtype=case["dtype"], device=DEVICE, source=DictSource(params), page_size=PAGE,
                                     max_total_tokens=held + PAGE, max_requests=case["requests"], max_tokens_per_step=PORTION)
    block = runner.model.blocks[0]
    state = {"runner": runner, "part": part}
    if part in ("mlp", "experts"):
        state["layer"], state["x"] = block.feed_forward, torch.cat(rows)
        return state
    slots = [runner.admit() for _ in past]
    todo, at = list(range(len(past))), [0] * len(past)
    while todo:                                     # the cached tokens, in prompt steps of at most PORTION tokens
        entries, xs, room = [], [], PORTION
        for i in list(todo):
            n = min(past[i] - at[i], room)
            if n > 0:
                part_of = rows[i][at[i]:at[i] + n]
                entries.append(StepEntry(slots[i], part_of.tolist() if part == "step" else [0] * n))
                xs.append(part_of)
                at[i], room = at[i] + n, room - n
            if at[i] == past[i]:
                todo.remove(i)
        if not entries:
            break
        if part == "step":
            runner.step(entries)
        else:
            batch = runner.prepare(entries)
            block.mixer.forward(torch.cat(xs), runner.model.stage_context(0, batch, runner.cache))
            runner.finish(batch)
    tails = [r[p:] for r, p in zip(rows, past)]
    entries = [StepEntry(s, t.tolist() if part == "step" else [0] * n, [n - 1] if part == "step" else [])
               for s, t, n in zip(slots, tails, new)]
    if part == "step":
        state["entries"] = entries
        return state
    batch = runner.prepare(entries)
    state.update(layer=block.mixer, x=torch.cat(tails), ctx=runner.model.stage_context(0, batch, runner.cache))
    return state


def _rest(config, weights, dtype):
    """`weights` beside the one-layer model's other tensors (embedding, norms, head), which the timed part does not read."""
    from litellmengine_b200.parts.model import model_parameters
    out = dict(weights)
    for name, spec in model_parameters(config.plan()).items():
        if name not in out and spec.optional_alias is None:
            out[name] = torch.ones(spec.shape, device=DEVICE, dtype=torch.float32 if spec.role == "scale" else dtype)
    return out


def run(state):
    part, runner = state["part"], state["runner"]
    if part == "step":                              # the step's position is not committed, so a pass is the same step again
        return {"logits": runner.forward(runner.prepare(state["entries"])), "kept": runner.cache.groups[0].kv}
    if part in ("mlp", "experts"):
        return state["layer"].forward(state["x"])
    ctx = state["ctx"]
    y = state["layer"].forward(state["x"], ctx)
    if part in ("gla", "delta"):
        return {"y": y, "kept": ctx.state}
    return {"y": y, "kept": ctx.cache if ctx.cache is not None else ctx.cache_keys}


# ---- what a pass cannot do without --------------------------------------------------------------------------
def _pairs(case, window=None, keep=0):
    total = 0
    for past, new in zip(_contexts(case), _portions(case)):
        i = np.arange(past, past + new, dtype=np.int64) + 1
        total += int(i.sum()) if window is None else int((np.minimum(i, window) + np.clip(i - window, 0, keep)).sum())
    return total


def _reach(case, window=None, keep=0):
    """Cached and new positions that some query of the step reads."""
    total = 0
    for past, new in zip(_contexts(case), _portions(case)):
        n = past + new
        total += n if window is None else min(n, new + window - 1 + keep)
    return total


def work(case):
    part, W, T = case["part"], case["width"], case["tokens"]
    ff, heads, kv = SIZES[W]
    es = 2 if case["dtype"] == "bfloat16" else 4
    matrices = {n: s[0] * s[1] for n, (s, k) in _shapes(case).items() if k == "matrix"}
    params = sum(matrices.values())
    if part == "step":
        heads, kv = QWEN_HEADS[W]
        body = sum(v for n, v in matrices.items() if n.startswith("model.layers."))
        head = STEP_VOCAB[W] * W
        kvb = 2 * kv * HEAD * es * _reach(case) * case["layers"]
        return {"bytes": (body + head) * es + kvb + T * STEP_VOCAB[W] * 4,
                "flops": 2 * T * (body + head) + 4 * heads * HEAD * _pairs(case) * case["layers"]}
    io = T * W * (es + 4)
    if part == "mlp":
        params = 3 * W * ff
        return {"bytes": params * es + io, "flops": 2 * T * params}
    if part == "experts":
        touched = min(EXPERTS, T * TOP)
        mine = 3 * W * (ff // 2)
        shared = 3 * W * (ff // 4)
        return {"bytes": (touched * mine + shared) * es + io, "flops": 2 * T * (TOP * mine + shared)}
    if part == "attention":
        heads, kv = QWEN_HEADS[W]
        params = W * HEAD * (2 * heads + 2 * kv)
        return {"bytes": params * es + io + 2 * kv * HEAD * es * _reach(case), "flops": 2 * T * params + 4 * heads * HEAD * _pairs(case)}
    if part == "windowed":
        return {"bytes": params * es + io + 2 * kv * HEAD * es * _reach(case, WINDOW, KEEP_FIRST),
                "flops": 2 * T * params + 4 * heads * HEAD * _pairs(case, WINDOW, KEEP_FIRST)}
    if part == "latent":
        row = LATENT_RANK + LATENT_ROT
        # per pair of a query and a key and per head: the score over key and rotated part, the value sum; the maps of the
        # latents are in the matrices, once per new token
        return {"bytes": params * es + io + row * es * _reach(case), "flops": 2 * T * params + 2 * heads * (2 * HEAD + LATENT_ROT) * _pairs(case)}
    half = max(1, heads // 2)
    state = case["requests"] * half * HEAD * HEAD * 4
    per_token = (5 if part == "gla" else 7) * half * HEAD * HEAD       # decay, write and read of the state (and its correction)
    return {"bytes": params * es + io + 2 * state, "flops": 2 * T * params + per_token * T}


# Between two correct implementations: 32-bit sums in another order, or 16-bit roundings of the activations between kernels
# (2^-9 each, a few of them in a row).  Each is about four times the distance to `exact` of the layer; a whole step's grows
# with the square root of the layers.
TOLERANCE = {"float32": {"step": 5e-5, "attention": 1e-5, "mlp": 1e-5},
             "bfloat16": {"step": 0.03, "attention": 0.015, "mlp": 0.012, "latent": 0.018, "gla": 0.007, "delta": 0.007,
                          "windowed": 0.014, "experts": 0.007}}


def tolerance(case):
    return {"rel": TOLERANCE[case["dtype"]][case["part"]], "max": 0.3 if case["dtype"] == "bfloat16" else 1e-3}


# ---- the same in 64 bits ------------------------------------------------------------------------------------
def _rms(x, eps, weight):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * weight


def _rotate(t, positions, base, dims, neighbours):
    """t [T, heads, n]: pairs (i, i + dims / 2), or (2i, 2i + 1), of the first `dims` entries turned by p * base^(-2i / dims)."""
    half = dims // 2
    f = base ** (-2.0 * torch.arange(half, dtype=F64, device=t.device) / dims)
    a = positions.to(F64)[:, None, None] * f
    c, s = torch.cos(a), torch.sin(a)
    out = t.clone()
    u, v = (slice(0, dims, 2), slice(1, dims, 2)) if neighbours else (slice(0, half), slice(half, dims))
    out[..., u] = t[..., u] * c - t[..., v] * s
    out[..., v] = t[..., v] * c + t[..., u] * s
    return out


def _softmax_over(q, k, v, scale, first, window=None, keep=0, sink=None):
    """q [T, H, D] at positions first .. first + T - 1, k [S, G, D], v [S, G, E] at 0 .. S - 1: [T, H, E]."""
    T, H, _ = q.shape
    rep, out = H // k.shape[1], torch.empty(T, H, v.shape[2], dtype=F64, device=q.device)
    kh, vh = k.permute(1, 2, 0), v.permute(1, 0, 2)
    j = torch.arange(k.shape[0], device=q.device)
    for at in range(0, T, 256):
        i = torch.arange(at, min(T, at + 256), device=q.device) + first
        qs = q[at:at + 256].permute(1, 0, 2).reshape(k.shape[1], -1, q.shape[2])
        s = (qs @ kh).view(H, len(i), -1) * scale
        seen = j <= i[:, None]
        if window is not None:
            seen &= (i[:, None] - j < window) | (j < keep)
        s = s.masked_fill(~seen, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(H, len(i), 1)], -1)
        p = torch.softmax(s, -1)
        p = p[..., :len(j)] if sink is not None else p
        out[at:at + 256] = (p.reshape(k.shape[1], rep * len(i), -1) @ vh).view(H, len(i), -1).permute(1, 0, 2)
    return out


def _qwen_attention(w, p, x, first, width):
    """x [S, W]: a whole sequence; the outputs of positions first .. S - 1."""
    heads, kv = QWEN_HEADS[width]
    S, g = x.shape[0], lambda n: w[p + n + ".weight"].to(F64)
    pos = torch.arange(S, device=x.device)
    q = _rotate(_rms((x[first:] @ g("q_proj").T).view(-1, heads, HEAD), EPS["qwen"], g("q_norm")), pos[first:], THETA, HEAD, False)
    k = _rotate(_rms((x @ g("k_proj").T).view(S, kv, HEAD), EPS["qwen"], g("k_norm")), pos, THETA, HEAD, False)
    v = (x @ g("v_proj").T).view(S, kv, HEAD)
    return _softmax_over(q, k, v, HEAD ** -0.5, first).reshape(S - first, -1) @ g("o_proj").T


def _qwen_mlp(w, p, x):
    g = lambda n: w[p + n + "_proj.weight"].to(F64)
    return (torch.nn.functional.silu(x @ g("gate").T) * (x @ g("up").T)) @ g("down").T


def _latent(w, x, first, width):
    heads = SIZES[width][1]
    S, R, P, g = x.shape[0], LATENT_RANK, LATENT_ROT, lambda n: w["l0.mix." + n].to(F64)
    pos, eps = torch.arange(S, device=x.device), EPS["design"]
    q = (_rms(x[first:] @ g("dq").T, eps, g("dq.norm")) @ g("uq").T).view(-1, heads, HEAD + P)
    q = torch.cat([q[..., :HEAD], _rotate(q[..., HEAD:], pos[first:], 10000.0, P, True)], -1)
    down = x @ g("dkv").T
    c = _rms(down[:, :R], eps, g("dkv.norm"))
    kr = _rotate(down[:, None, R:], pos, 10000.0, P, True).expand(S, heads, P)
    k = torch.cat([(c @ g("uk").T).view(S, heads, HEAD), kr], -1)
    o = _softmax_over(q, k, (c @ g("uv").T).view(S, heads, HEAD), (HEAD + P) ** -0.5, first)
    return (o * torch.sigmoid(x[first:] @ g("g").T)[:, :, None]).reshape(S - first, -1) @ g("o").T


def _windowed(w, x, first, width):
    _, heads, kv = SIZES[width]
    S, g = x.shape[0], lambda n: w["l0.mix." + n].to(F64)
    pos = torch.arange(S, device=x.device)
    q = _rotate((x[first:] @ g("q").T).view(-1, heads, HEAD), pos[first:], 10000.0, LATENT_ROT, False)
    k = _rotate((x @ g("k").T).view(S, kv, HEAD), pos, 10000.0, LATENT_ROT, False)
    o = _softmax_over(q, k, (x @ g("v").T).view(S, kv, HEAD), HEAD ** -0.5, first, WINDOW, KEEP_FIRST, g("sink"))
    return o.reshape(S - first, -1) @ g("o").T


def _gla(w, x, first, width):
    half, eps = max(1, SIZES[width][1] // 2), EPS["design"]
    T, g = x.shape[0], lambda n: w["l0.mix." + n].to(F64)
    split = lambda n: (x @ g(n).T).view(T, half, HEAD)
    q, k, v = split("q") * HEAD ** -0.5, split("k"), split("v")
    decay = torch.exp(torch.nn.functional.logsigmoid((x @ g("a1").T) @ g("a2").T + g("a2.b")) / TAU).view(T, half, HEAD)
    S, o = torch.zeros(half, HEAD, HEAD, dtype=F64, device=x.device), torch.empty(T, half, HEAD, dtype=F64, device=x.device)
    for t in range(T):
        S = torch.baddbmm(decay[t][:, :, None] * S, k[t][:, :, None], v[t][:, None, :])
        o[t] = (q[t][:, None, :] @ S)[:, 0]
    o = _rms(o, eps, g("norm")).reshape(T, -1) * torch.nn.functional.silu(x @ g("g").T)
    return o[first:] @ g("o").T, S


def _delta(w, x, first, width):
    half, eps = max(1, SIZES[width][1] // 2), EPS["design"]
    T, g = x.shape[0], lambda n: w["l0.mix." + n].to(F64)

    def conv(n):
        u, taps, out = x @ g(n).T, g(n + ".conv"), 0.0
        for j in range(TAPS):
            back = TAPS - 1 - j
            out = out + torch.nn.functional.pad(u, (0, 0, back, 0))[:T] * taps[:, j]
        return torch.nn.functional.silu(out).view(T, half, HEAD)
    unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
    q, k, v = unit(conv("q")) * HEAD ** -0.5, unit(conv("k")), conv("v")
    beta = torch.sigmoid(x @ g("b").T)
    z = (x @ g("a1").T) @ g("a2").T + g("dt_bias")
    decay = torch.exp(-torch.exp(g("A_log"))[None, :, None] * torch.nn.functional.softplus(z).view(T, half, HEAD))
    S, o = torch.zeros(half, HEAD, HEAD, dtype=F64, device=x.device), torch.empty(T, half, HEAD, dtype=F64, device=x.device)
    for t in range(T):
        S = decay[t][:, :, None] * S
        write = beta[t][:, None, None] * (v[t][:, None, :] - k[t][:, None, :] @ S)
        S = torch.baddbmm(S, k[t][:, :, None], write)
        o[t] = (q[t][:, None, :] @ S)[:, 0]
    o = _rms(o, eps, g("norm")).reshape(T, -1) * torch.sigmoid((x @ g("g1").T) @ g("g2").T)
    return o[first:] @ g("o").T


def _experts(w, x):
    g = lambda n: w["l0.mlp." + n].to(F64)

    def expert(e, t):
        a, b = torch.clamp(t @ g(e + "gate").T, max=LIMIT), torch.clamp(t @ g(e + "up").T, -LIMIT, LIMIT)
        return (a * torch.sigmoid(1.702 * a) * (b + 1.0)) @ g(e + "down").T
    best = torch.topk(x @ g("router").T + g("router.b"), TOP, dim=-1)
    share = torch.softmax(best.values, -1)
    out = torch.sigmoid(x @ g("shared.sg").T) * expert("shared.", x)
    for e in range(EXPERTS):
        row, place = (best.indices == e).nonzero(as_tuple=True)
        out[row] += share[row, place][:, None] * expert(f"e{e}.", x[row])
    return out


def exact(case, seed):
    part, W = case["part"], case["width"]
    w, past = _weights(case, seed), _contexts(case)
    if part in ("gla", "delta") and sum(past) + case["tokens"] > 12000:
        return None                                 # token by token: too long a walk
    rows = _rows(case, seed)
    if part == "step":
        out = []
        for ids in rows:
            x = w["model.embed_tokens.weight"][ids].to(F64)
            for i in range(case["layers"]):
                p = f"model.layers.{i}."
                n = lambda name: w[p + name + "_layernorm.weight"].to(F64)
                x = x + _qwen_attention(w, p + "self_attn.", _rms(x, EPS["qwen"], n("input")), 0, W)
                x = x + _qwen_mlp(w, p + "mlp.", _rms(x, EPS["qwen"], n("post_attention")))
            head = w["model.embed_tokens.weight" if W == 1024 else "lm_head.weight"].to(F64)
            out.append(_rms(x[-1:], EPS["qwen"], w["model.norm.weight"].to(F64)) @ head.T)
        return {"logits": torch.cat(out), "kept": None}
    if part == "mlp":
        return _qwen_mlp(w, "model.layers.0.mlp.", torch.cat(rows).to(F64))
    if part == "experts":
        return _experts(w, torch.cat(rows).to(F64))
    of = {"attention": lambda x, f: _qwen_attention(w, "model.layers.0.self_attn.", x, f, W), "latent": lambda x, f: _latent(w, x, f, W),
          "windowed": lambda x, f: _windowed(w, x, f, W), "gla": lambda x, f: _gla(w, x, f, W), "delta": lambda x, f: _delta(w, x, f, W)}[part]
    got = [of(x.to(F64), f) for x, f in zip(rows, past)]
    if part == "gla":
        return {"y": torch.cat([y for y, _ in got]), "kept": torch.stack([s for _, s in got])}
    return {"y": torch.cat(got), "kept": None}
