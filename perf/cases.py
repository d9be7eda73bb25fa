"""Timed cases: what a user of this engine has it do, through its public entry points.

Two whole calls (`ModelRunner.step`: a decode step and a step of prompts, with logits) and the layers' parts one by one
(`Mixer.forward`, `FeedForward.forward`), at the layer sizes of the Qwen2.5-1.5B and 7B shapes and of the other designs at
those sizes, as in bench.py.  `draw` varies every one of them: requests, tokens, contexts, sizes, kinds of part.

A case is a dict of numbers and texts.  How its tokens fall on its requests, and how much context each of them has, follows
from the case alone; weights, inputs and cached context follow from the seed.
"""
from __future__ import annotations

import math
import random

import torch
import torch.nn.functional as F

from inferflux_b200.cache import CacheManager
from inferflux_b200.config import PartSpec, Qwen2Config, ScheduleEntry
from inferflux_b200.csrc import CudaKernels
from inferflux_b200.engine import ModelRunner, StepContext, StepEntry
from inferflux_b200.models.model import Model
from inferflux_b200.parts import build_part

DEV = "cuda:0"
PAGE = 16
EPS = 1e-6
THETA = 1e6
# width, feed-forward size, query heads, key/value heads, vocabulary
SHAPES = {"1.5b": (1536, 8960, 12, 2, 151936), "7b": (3584, 18944, 28, 4, 152064)}
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
MIXERS = ("wkv", "delta_rule", "decayed_linear_attention", "state_space", "retention", "lightning")


def listed():
    return [
        # a decode step of a served model: eight requests at a context of a few thousand tokens, logits for the next token of
        # each; four layers of the 7B shape stand for its 28
        {"name": "decode_step", "kind": "decode_step", "shape": "7b", "layers": 4, "requests": 8, "context": 2048},
        # a step in which several prompts arrive: chunked prefill of about 1,500 tokens, logits of every prompt's last token
        {"name": "prompt_step", "kind": "prompt_step", "shape": "1.5b", "layers": 8, "requests": 3, "tokens": 1531},
        # the smallest call: one token of one chat through a feed-forward (weights read once, launches count)
        {"name": "mlp_one_token", "kind": "mlp", "shape": "1.5b", "rows": 1, "dtype": "bfloat16"},
        # the 32-bit run (exactness checks, trace replay), a prompt portion through a feed-forward
        {"name": "mlp_float32", "kind": "mlp", "shape": "1.5b", "rows": 333, "dtype": "float32"},
        # attention layer, prompts: portions of two long documents, one of them with thousands of tokens before it
        {"name": "attention_prompt", "kind": "attention", "shape": "7b", "requests": 2, "tokens": 2500, "context": 4000},
        # attention layer, decoding: 64 requests of mixed lengths
        {"name": "attention_decode", "kind": "attention", "shape": "7b", "requests": 64, "tokens": 64, "context": 8000},
        # latent attention layer with a rotated key part and queries through a latent of their own: a prompt portion
        {"name": "latent_prompt", "kind": "latent", "shape": "1.5b", "rot": 64, "requests": 1, "tokens": 2048, "context": 0},
        # the same, decoding at the long contexts that small cached rows are for
        {"name": "latent_decode", "kind": "latent", "shape": "1.5b", "rot": 64, "requests": 64, "tokens": 64, "context": 16000},
        # a mixture of 16 gated experts, four of which a token uses: a decode batch, and a prompt portion through plain experts
        # two of whose router outputs hand the token on unchanged
        {"name": "moe_decode", "kind": "moe", "shape": "1.5b", "glu": 1, "rows": 24},
        {"name": "moe_prompt", "kind": "moe", "shape": "1.5b", "glu": 0, "rows": 2048},
        # layers with a matrix of state per head instead of a cache: a prompt portion (delta rule), two prompts (constant decay)
        {"name": "delta_prompt", "kind": "recurrent", "mixer": "delta_rule", "shape": "1.5b", "requests": 1, "tokens": 2048},
        {"name": "lightning_prompt", "kind": "recurrent", "mixer": "lightning", "shape": "1.5b", "requests": 2, "tokens": 1901},
    ]


def draw(rng):
    """One more case of the listed ones' ranges."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["decode_step", "prompt_step", "mlp", "mlp", "attention_prompt", "attention_decode", "latent_prompt",
                       "latent_decode", "moe", "moe", "recurrent", "recurrent"])
    shape = rng.choice(list(SHAPES))
    if kind == "decode_step":
        return {"kind": kind, "shape": shape, "layers": rng.randint(2, 4), "requests": log_int(1, 48),
                "context": log_int(64, 2048)}
    if kind == "prompt_step":
        return {"kind": kind, "shape": "1.5b", "layers": rng.randint(2, 8), "requests": rng.randint(1, 6),
                "tokens": log_int(100, 1500)}
    if kind == "mlp":
        dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
        return {"kind": kind, "shape": shape, "rows": log_int(1, 1000 if dtype == "bfloat16" else 300), "dtype": dtype}
    if kind == "attention_prompt":
        return {"kind": "attention", "shape": shape, "requests": rng.randint(1, 5), "tokens": log_int(60, 2500),
                "context": rng.choice([0, log_int(100, 4000)])}
    if kind == "attention_decode":
        n = log_int(1, 64)
        return {"kind": "attention", "shape": shape, "requests": n, "tokens": n, "context": log_int(200, 8000)}
    if kind == "latent_prompt":
        return {"kind": "latent", "shape": shape, "rot": rng.choice([0, 64]), "requests": rng.randint(1, 4),
                "tokens": log_int(60, 2048 if shape == "1.5b" else 1200), "context": rng.choice([0, log_int(100, 2000)])}
    if kind == "latent_decode":
        n = log_int(1, 64)
        return {"kind": "latent", "shape": shape, "rot": rng.choice([0, 64]), "requests": n, "tokens": n,
                "context": log_int(400, 16000)}
    if kind == "moe":
        return {"kind": kind, "shape": shape, "glu": rng.randint(0, 1), "rows": log_int(1, 2048 if shape == "1.5b" else 700)}
    n = rng.randint(1, 4)
    return {"kind": kind, "mixer": rng.choice(MIXERS), "shape": shape, "requests": n,
            "tokens": log_int(max(40, n), 2048 if shape == "1.5b" else 1500)}


# ------------------------------------------------------------------------------- what a case consists of
def _spans(case):
    """(tokens of context, new tokens) of every request: uneven shares, the same for every seed."""
    n, total, context = case["requests"], case.get("tokens", case["requests"]), case.get("context", 0)
    r = random.Random(1000003 * n + 1009 * total + context)
    weights = [r.uniform(0.3, 1.7) for _ in range(n)]
    spans, left = [], total - n
    for i in range(n):
        extra = left if i == n - 1 else min(left, int((total - n) * weights[i] / sum(weights)))
        left -= extra
        spans.append(1 + extra)
    return [(int(context * r.uniform(0.1, 1.0)), s) for s in spans]


def _model_config(case):
    width, inter, heads, kv_heads, vocab = SHAPES[case["shape"]]
    return Qwen2Config(hidden_size=width, num_hidden_layers=case["layers"], num_attention_heads=heads,
                       num_key_value_heads=kv_heads, head_dim=128, intermediate_size=inter, vocab_size=vocab,
                       max_position_embeddings=32768, rope_theta=THETA, rms_norm_eps=EPS, tie_word_embeddings=False)


def _part_spec(case):
    """(role, PartSpec) of a part's case."""
    width, inter, heads, kv_heads, _ = SHAPES[case["shape"]]
    kind = case["kind"]
    if kind == "mlp":
        return "ffn", PartSpec("swiglu", {"hidden_size": width, "intermediate_size": inter})
    if kind == "attention":
        return "mixer", PartSpec("attention", {
            "hidden_size": width, "num_heads": heads, "num_kv_heads": kv_heads, "head_dim": 128, "window": None, "scale": None,
            "qkv_bias": True, "position": PartSpec("rope", {"theta": THETA, "rotary_dim": 128, "pairing": "split_half"})})
    if kind == "latent":
        params = {"hidden_size": width, "num_heads": heads, "qk_dim": 128, "v_dim": 128, "kv_rank": 256,
                  "scale": (128 + case["rot"]) ** -0.5}
        if case["rot"]:
            params.update({"q_rank": 1536, "rot_dim": case["rot"], "position": PartSpec(
                "rope", {"theta": THETA, "rotary_dim": case["rot"], "pairing": "interleaved"})})
        return "mixer", PartSpec("latent_attention", params)
    if kind == "moe":
        params = {"hidden_size": width, "num_experts": 16, "top": 4}
        if case["glu"]:
            params.update({"expert_size": (inter // 4) // 64 * 64, "activation": "clamped_glu", "limit": 7.0,
                           "routing": "softmax_of_chosen", "correction": False})
        else:
            params.update({"expert_size": (3 * inter // 8) // 64 * 64, "num_identity": 2})
        return "ffn", PartSpec("moe", params)
    mixer = case["mixer"]
    if mixer in ("wkv", "delta_rule"):
        params = {"num_heads": width // 64, "head_dim": 64, "decay_rank": 64}
    elif mixer == "decayed_linear_attention":
        params = {"num_heads": width // 128, "key_dim": 64, "value_dim": 128, "tau": 16.0, "decay_rank": 16}
    elif mixer == "state_space":
        params = {"num_heads": width // 64, "value_dim": 64, "state_dim": 128, "groups": 1, "conv_taps": 4}
    else:
        h = width // 128
        params = {"num_heads": h, "key_dim": 64 if mixer == "retention" else 128, "value_dim": 128,
                  "decay": [1.0 - 2.0 ** (-5.0 - 5.0 * i / h) for i in range(h)]}
        if mixer == "retention":
            params["position"] = PartSpec("rope", {"theta": 1e4, "rotary_dim": 64, "pairing": "split_half"})
    return "mixer", PartSpec(mixer, {"hidden_size": width, "norm_eps": EPS, **params})


# where a recurrence's parameters lie in trained models: memories from a few tokens to thousands
_RANGES = {"wkv": {"w0": (-6.0, -0.5)}, "delta_rule": {"w0": (-6.0, 1.0)},
           "decayed_linear_attention": {"a2.b": (-2.0, 4.0)}, "state_space": {"A_log": (0.0, 2.7), "dt_bias": (-6.0, -2.0)}}


def _tensors(specs, dtype, seed, ranges=None):
    """Weights by name: N(0, 0.02) matrices, norms near one, other vectors spread about zero."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    out = {}
    for name in sorted(specs):
        spec = specs[name]
        shape = spec.shape_to_make()
        if ranges and name in ranges:
            lo, hi = ranges[name]
            out[name] = torch.rand(shape, generator=g, device=DEV) * (hi - lo) + lo
        elif spec.init == "ones":
            out[name] = 1 + 0.1 * torch.randn(shape, generator=g, device=DEV)
        elif spec.init == "zeros" or len(shape) == 1:
            out[name] = torch.rand(shape, generator=g, device=DEV) * (0.5 if spec.init == "zeros" else 0.2)
        elif shape[-1] <= 16:                                 # taps of a convolution
            out[name] = 0.3 * torch.randn(shape, generator=g, device=DEV)
        else:
            out[name] = (0.02 * torch.randn(shape, generator=g, device=DEV)).to(dtype)
    return out


def _rows(case, dtype, seed):
    """The layer's input: rows behind a norm, or the float32 stream."""
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    total = case["rows"] if "rows" in case else sum(n for _, n in _spans(case))
    return torch.randn(total, SHAPES[case["shape"]][0], generator=g, device=DEV).to(dtype)


def _context_rows(shape, seed, r):
    g = torch.Generator(device=DEV).manual_seed(seed + 17 + r)
    return torch.randn(shape, generator=g, device=DEV).to(torch.bfloat16)


_KERNELS = []


def _kernels():
    """The kernel table, one for the process, as in any program."""
    if not _KERNELS:
        _KERNELS.append(CudaKernels(DEV))
    return _KERNELS[0]


class _FeedForwardContext:
    def __init__(self, kernels, dtype):
        self.kernels, self.dtype = kernels, dtype


# ------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    if case["kind"] in ("decode_step", "prompt_step"):
        return _prepare_step(case, seed)
    dtype = DTYPES[case.get("dtype", "bfloat16")]
    role, spec = _part_spec(case)
    part = build_part(role, spec)
    part.load(_tensors(part.param_specs(), dtype, seed, _RANGES.get(spec.kind)), dtype, DEV)
    kernels = _kernels()
    state = {"part": part, "h": _rows(case, torch.float32 if part.takes_stream else dtype, seed)}
    if role == "ffn":
        state["ctx"] = _FeedForwardContext(kernels, dtype)
        return state
    spans = _spans(case)
    longest = max(c + n for c, n in spans)
    pages = sum(-(-(c + n) // PAGE) for c, n in spans)
    cache = CacheManager([(part.cache_spec(), part.state_spec())], page_size=PAGE, num_pages=pages, max_seqs=len(spans),
                         max_seq_len=longest, dtype=dtype, device=DEV)
    view = cache.view(ScheduleEntry(0, 0))
    for r, (c, n) in enumerate(spans):                         # request r has slot r
        cache.add_request(r)
        cache.reserve(r, c + n)
        if c and view.kv is not None:                          # what earlier steps stored
            held = cache.pages_of(r)
            _, planes, heads, page, d = view.kv.shape
            blocks = -(-c // page)
            rows = _context_rows((blocks, planes, heads, page, d), seed, r)
            view.kv[torch.tensor([held[b] for b in range(blocks)], device=DEV)] = rows
    ctx = StepContext.build(kernels, dtype, DEV, [StepEntry(r, [0] * n, []) for r, (_, n) in enumerate(spans)],
                            [c for c, _ in spans], [cache.slot(r) for r in range(len(spans))], cache.drain_table_updates(),
                            providers=[part])
    for group, (index, page_id) in zip(cache.groups, ctx.table_updates):
        kernels.scatter_i32(group.table, index, page_id)
    state.update({"ctx": ctx, "cache": view, "manager": cache})
    return state


def _prepare_step(case, seed):
    cfg = _model_config(case)
    model = Model(cfg.to_plan())
    specs = {n: s for n, s in model.expected_tensors().items() if not s.ignored}
    model.load(_tensors(specs, torch.bfloat16, seed), torch.bfloat16, DEV)
    spans = _spans(case)
    prompts = _token_ids(case, seed)
    if case["kind"] == "prompt_step":
        runner = ModelRunner(model, _kernels(), page_size=PAGE, num_pages=sum(-(-n // PAGE) for _, n in spans),
                             max_seqs=len(spans), max_seq_len=max(n for _, n in spans))
        return {"runner": runner, "end": True,
                "entries": [StepEntry(r, p, [len(p) - 1]) for r, p in enumerate(prompts)]}
    room = 8192                                                # steps that the cache can still take
    runner = ModelRunner(model, _kernels(), page_size=PAGE, num_pages=sum(-(-(c + room) // PAGE) for c, _ in spans),
                         max_seqs=len(spans), max_seq_len=case["context"] + room, cuda_graphs=True)
    for r, p in enumerate(prompts):
        if len(p) > 1:
            runner.step([StepEntry(r, p[:-1], [])])
    return {"runner": runner, "end": False, "entries": [StepEntry(r, p[-1:], [0]) for r, p in enumerate(prompts)]}


def _token_ids(case, seed):
    r = random.Random(seed)
    vocab = SHAPES[case["shape"]][4]
    return [[r.randrange(vocab) for _ in range(c + n)] for c, n in _spans(case)]


def run(state):
    if "runner" in state:
        logits = state["runner"].step(state["entries"])
        if state["end"]:
            for e in state["entries"]:
                state["runner"].end_request(e.request_id)
        return {"logits": logits}
    ctx, part = state["ctx"], state["part"]
    if "cache" not in state:
        return {"y": ctx.kernels.materialize(part.forward(state["h"], ctx))}
    y = ctx.kernels.materialize(part.forward(state["h"], ctx, state["cache"]))
    cache = state["cache"]
    out = {"y": y}
    if cache.state is not None:
        out["state"] = cache.state
    if cache.kv is not None:
        out["cache"] = cache.kv
    return out


# ------------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    width, inter, heads, kv_heads, vocab = SHAPES[case["shape"]]
    kind = case["kind"]
    spans = None if "rows" in case else _spans(case)
    rows = case["rows"] if "rows" in case else sum(n for _, n in spans)
    qkv = (heads + 2 * kv_heads) * 128 * width
    o = heads * 128 * width
    if kind in ("decode_step", "prompt_step"):
        layer = qkv + o + 3 * width * inter
        head = vocab * width
        seen = sum(c + n for c, n in spans)
        pairs = sum(n * c + n * (n + 1) // 2 for c, n in spans)
        return {"bytes": 2 * (case["layers"] * layer + head) + case["layers"] * seen * 4 * kv_heads * 128
                + rows * width * 2 + len(spans) * vocab * 4,
                "flops": 2 * rows * case["layers"] * layer + 2 * len(spans) * head + case["layers"] * 4 * heads * 128 * pairs}
    size = 4 if case.get("dtype") == "float32" else 2
    if kind == "mlp":
        return {"bytes": size * (3 * width * inter + 2 * rows * width), "flops": 2 * rows * 3 * width * inter}
    if kind == "moe":
        ff = (inter // 4) // 64 * 64 if case["glu"] else (3 * inter // 8) // 64 * 64
        expert = (3 if case["glu"] else 2) * ff * width
        share = 4.0 if case["glu"] else 4.0 * 16 / 18           # choices of a token that have weights
        used = 16 * (1 - (1 - share / 16) ** rows)               # experts that some token chooses
        return {"bytes": 2 * (used * expert + (16 if case["glu"] else 18) * width + 2 * rows * width),
                "flops": 2 * rows * share * expert}
    pairs = sum(n * c + n * (n + 1) // 2 for c, n in spans)
    seen = sum(c + n for c, n in spans)
    if kind == "attention":
        return {"bytes": 2 * (qkv + o) + seen * 4 * kv_heads * 128 + rows * width * 4,
                "flops": 2 * rows * (qkv + o) + 4 * heads * 128 * pairs}
    if kind == "latent":
        rot = case["rot"]
        q = width * 1536 + 1536 * heads * (128 + rot) if rot else width * heads * 128
        weights = q + width * (256 + rot) + 2 * heads * 128 * 256 + o
        # decoded tokens meet the latents as they are, prompts could meet keys and values made from them
        per_pair = 2 * heads * ((256 + rot) + 256) if rows == len(spans) else 2 * heads * ((128 + rot) + 128)
        return {"bytes": 2 * weights + seen * 2 * (256 + rot) + rows * width * 4, "flops": 2 * rows * weights + per_pair * pairs}
    h, dk, dv, proj = _recurrent_sizes(case)
    return {"bytes": 2 * proj + rows * width * (8 if case["mixer"] in ("wkv", "decayed_linear_attention", "state_space") else 4)
            + 2 * len(spans) * h * dk * dv * 4,
            "flops": 2 * rows * proj + 4 * rows * h * dk * dv}


def _recurrent_sizes(case):
    """heads, key channels, value channels, numbers in the projections."""
    w, mixer = SHAPES[case["shape"]][0], case["mixer"]
    if mixer == "wkv":
        return w // 64, 64, 64, 5 * w * w + 2 * 64 * w
    if mixer == "delta_rule":
        return w // 64, 64, 64, 6 * w * w + 2 * 64 * w
    if mixer == "decayed_linear_attention":
        return w // 128, 64, 128, 4 * w * w + 16 * w + 8 * w
    if mixer == "state_space":
        return w // 64, 128, 64, w * (2 * w + 256 + w // 64) + w * w
    if mixer == "retention":
        return w // 128, 64, 128, 4 * w * w
    return w // 128, 128, 128, 5 * w * w


def tolerance(case):
    """Relative errors that the data types bring: about four times what a run shows against `exact`."""
    kind = case["kind"]
    if case.get("dtype") == "float32":
        return {"rel": 8e-6}
    if kind in ("decode_step", "prompt_step"):                   # every layer's rounding travels through those that follow
        return {"rel": 0.03, "max": 0.5}
    return {"rel": 0.02 if kind in ("attention", "latent") else 0.01, "max": 0.4}


# ------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode_step", "prompt_step"):
        return {"logits": _exact_logits(case, seed)}
    dtype = DTYPES[case.get("dtype", "bfloat16")]
    role, spec = _part_spec(case)
    part = build_part(role, spec)                               # for the names and shapes of its tensors alone
    w = {n: t.double() for n, t in _tensors(part.param_specs(), dtype, seed, _RANGES.get(spec.kind)).items()}
    x = _rows(case, torch.float32 if part.takes_stream else dtype, seed).double()
    if kind == "mlp":
        return {"y": (F.silu(x @ w["gate_proj.weight"].T) * (x @ w["up_proj.weight"].T)) @ w["down_proj.weight"].T}
    if kind == "moe":
        return {"y": _exact_moe(case, x, w)}
    if kind == "attention":
        return {"y": _exact_attention(case, seed, x, w), "cache": None}
    if kind == "latent":
        return {"y": _exact_latent(case, seed, x, w), "cache": None}
    y, state = _exact_recurrent(case, spec.params, x, w)
    return {"y": y, "state": state}


def _rms(x, weight=None):
    y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)
    return y if weight is None else y * weight


def _rotate(x, positions, theta, interleaved=False):
    """Pairs of the last dimension of x [T, heads, d] turned by position * theta^(-2 i / d)."""
    d = x.shape[-1]
    freq = theta ** (-torch.arange(0, d, 2, dtype=torch.float64, device=x.device) / d)
    ang = (positions.double()[:, None] * freq)[:, None, :]
    cos, sin = ang.cos(), ang.sin()
    a, b = (x[..., 0::2], x[..., 1::2]) if interleaved else (x[..., :d // 2], x[..., d // 2:])
    lo, hi = a * cos - b * sin, b * cos + a * sin
    return torch.stack((lo, hi), -1).flatten(-2) if interleaved else torch.cat((lo, hi), -1)


def _attend(q, k, v, first, scale):
    """q [n, heads, d] at positions first .. over k, v [keys, kv heads, .]: causal, heads in groups."""
    n, heads, _ = q.shape
    group = heads // k.shape[1]
    keys = torch.arange(k.shape[0], device=q.device)
    out = torch.empty(n, heads, v.shape[-1], dtype=q.dtype, device=q.device)
    for t0 in range(0, n, 512):
        hidden = keys[None, :] > (first + t0 + torch.arange(min(512, n - t0), device=q.device))[:, None]
        for h in range(heads):
            s = q[t0:t0 + 512, h] @ k[:, h // group].T * scale
            out[t0:t0 + 512, h] = s.masked_fill(hidden, float("-inf")).softmax(-1) @ v[:, h // group]
    return out


def _exact_attention(case, seed, x, w):
    _, _, heads, kv_heads, _ = SHAPES[case["shape"]]
    q, k, v = (x @ w[f"{s}_proj.weight"].T + w[f"{s}_proj.bias"] for s in "qkv")
    out, at = [], 0
    for r, (c, n) in enumerate(_spans(case)):
        pos = torch.arange(c, c + n, device=DEV)
        qr = _rotate(q[at:at + n].view(n, heads, 128), pos, THETA)
        kr = _rotate(k[at:at + n].view(n, kv_heads, 128), pos, THETA)
        vr = v[at:at + n].view(n, kv_heads, 128)
        if c:
            rows = _context_rows((-(-c // PAGE), 2, kv_heads, PAGE, 128), seed, r).double()
            old = rows.permute(1, 0, 3, 2, 4).reshape(2, -1, kv_heads, 128)[:, :c]
            kr, vr = torch.cat((old[0], kr)), torch.cat((old[1], vr))
        out.append(_attend(qr, kr, vr, c, 128 ** -0.5).reshape(n, -1))
        at += n
    return torch.cat(out) @ w["o_proj.weight"].T


def _exact_latent(case, seed, x, w):
    heads, rot = SHAPES[case["shape"]][2], case["rot"]
    T = x.shape[0]
    q = x @ w["q"].T if not rot else _rms(x @ w["dq"].T, w["dq.norm"]) @ w["uq"].T
    q = q.view(T, heads, 128 + rot)
    down = x @ w["dkv"].T
    c_new = _rms(down[:, :256], w["dkv.norm"])
    uk, uv = w["uk"].view(heads, 128, 256), w["uv"].view(heads, 128, 256)
    ql = torch.einsum("thd,hdr->thr", q[..., :128], uk)
    out, at = [], 0
    for r, (c, n) in enumerate(_spans(case)):
        pos = torch.arange(c, c + n, device=DEV)
        keys, qr = c_new[at:at + n], ql[at:at + n]
        if rot:
            keys = torch.cat((keys, _rotate(down[at:at + n, None, 256:], pos, THETA, interleaved=True)[:, 0]), -1)
            qr = torch.cat((qr, _rotate(q[at:at + n, :, 128:], pos, THETA, interleaved=True)), -1)
        if c:
            old = _context_rows((-(-c // PAGE), 1, 1, PAGE, 256 + rot), seed, r).double().reshape(-1, 256 + rot)[:c]
            keys = torch.cat((old, keys))
        out.append(_attend(qr, keys[:, None], keys[:, None, :256], c, (128 + rot) ** -0.5))
        at += n
    return torch.einsum("thr,hvr->thv", torch.cat(out), uv).reshape(T, -1) @ w["o"].T


def _exact_moe(case, x, w):
    z = x @ w["router"].T
    if case["glu"]:
        chosen = z.topk(4, -1)
        ids, weights = chosen.indices, chosen.values.softmax(-1)
    else:
        scores = z.softmax(-1)
        ids = (scores + w["correction"].double()).topk(4, -1).indices
        weights = scores.gather(-1, ids)
    y = torch.zeros_like(x)
    for e in range(16 if case["glu"] else 18):
        hit, slot = (ids == e).nonzero(as_tuple=True)
        if not len(hit):
            continue
        h = x[hit]
        if e < 16:
            up = h @ w[f"e{e}.up"].T
            if case["glu"]:
                gate = (h @ w[f"e{e}.gate"].T).clamp(max=7.0)
                up = gate * torch.sigmoid(1.702 * gate) * (up.clamp(-7.0, 7.0) + 1)
            else:
                up = up.relu().square()
            h = up @ w[f"e{e}.down"].T
        y.index_add_(0, hit, h * weights[hit, slot, None])
    return y


def _exact_recurrent(case, p, x, w):
    mixer, spans = case["mixer"], _spans(case)
    heads, dk, dv, _ = _recurrent_sizes(case)
    T, hk = x.shape[0], heads * dk
    starts = [sum(n for _, n in spans[:i]) for i in range(len(spans))]

    def split(t, d):
        return t.view(T, heads, d)

    erase = unit = tail = None
    bonus = skip = 0.0
    if mixer == "wkv":
        before = x.roll(1, 0)
        before[starts] = 0
        mix = {s: x + (before - x) * w["mu." + s] for s in "rkvgw"}
        q, k, v, g = (mix[s] @ w[s].T for s in "rkvg")
        decay = torch.exp(-torch.exp(torch.tanh(mix["w"] @ w["w1"].T) @ w["w2"].T + w["w0"]))
        q, k, v, decay = split(q, dk), split(k, dk), split(v, dv), split(decay, dk)
        bonus = (q * w["u"] * k).sum(-1, keepdim=True) * v
        tail = torch.stack([x[s + n - 1] for s, (_, n) in zip(starts, spans)])
    elif mixer == "delta_rule":
        q, k, v, g, a = (x @ w[s].T for s in "rkvga")
        low = torch.tanh(x @ w["w1"].T) @ w["w2"].T + w["w0"]
        decay = split(torch.exp(-math.exp(-0.5) * torch.sigmoid(low)), dk)
        q, k, v = split(q, dk), split(k, dk), split(v, dv)
        unit = k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)
        erase = split(torch.sigmoid(a + w["a.b"]), dk) * unit
    elif mixer == "state_space":
        inner = heads * dv
        zx = x @ w["in"].T
        g, xbc, dt = zx[:, :inner], zx[:, inner:inner + inner + 2 * dk], zx[:, inner + inner + 2 * dk:]
        tail = torch.stack([F.pad(xbc[s:s + n], (0, 0, 3, 0))[-3:].flatten() for s, (_, n) in zip(starts, spans)])
        conv = torch.cat([sum(F.pad(xbc[s:s + n], (0, 0, 3, 0))[j:j + n] * w["conv"][:, j] for j in range(4))
                          for s, (_, n) in zip(starts, spans)])
        xbc = F.silu(conv + w["conv.b"])
        dt = F.softplus(dt + w["dt_bias"])
        v = split(xbc[:, :inner], dv)
        k = xbc[:, inner:inner + dk][:, None] * dt[..., None]
        q = xbc[:, inner + dk:][:, None].expand(T, heads, dk)
        decay = torch.exp(-torch.exp(w["A_log"]) * dt)[..., None].expand(T, heads, dk)
        skip = w["D"][:, None] * v
    else:
        act = F.silu if mixer == "lightning" else (lambda t: t)
        q, k, v = split(act(x @ w["q"].T), dk), split(act(x @ w["k"].T), dk), split(act(x @ w["v"].T), dv)
        g = x @ w["g"].T
        if mixer == "decayed_linear_attention":
            q = q * dk ** -0.5
            decay = split(torch.sigmoid(x @ w["a1"].T @ w["a2"].T + w["a2.b"]) ** (1 / p["tau"]), dk)
        else:
            if mixer == "retention":
                pos = torch.cat([torch.arange(n, device=DEV) for _, n in spans])
                q, k = _rotate(q, pos, 1e4), _rotate(k, pos, 1e4) * dk ** -0.5
            decay = torch.tensor(p["decay"], dtype=torch.float64, device=DEV)[:, None].expand(T, heads, dk)
    out = torch.empty(T, heads, dv, dtype=torch.float64, device=DEV)
    states = []
    for s, (_, n) in zip(starts, spans):
        S = torch.zeros(heads, dk, dv, dtype=torch.float64, device=DEV)
        for t in range(s, s + n):
            if mixer == "wkv":
                out[t] = (q[t, :, None] @ S)[:, 0]
            erased = 0.0 if unit is None else erase[t, :, :, None] * (unit[t, :, None] @ S)
            S = decay[t, :, :, None] * S - erased + k[t, :, :, None] * v[t, :, None]
            if mixer != "wkv":
                out[t] = (q[t, :, None] @ S)[:, 0]
        states.append(S)
    out = out + bonus + skip
    S = torch.stack(states)
    if mixer in ("wkv", "delta_rule"):
        state = S.flatten(1)
        gate = F.silu(g) if mixer == "wkv" else torch.sigmoid(g)
        y = _rms(out).reshape(T, -1) * w["norm"] * gate
    else:
        state = S.transpose(-1, -2).flatten(1)                   # [head, value channel, key channel]
        if mixer == "state_space":
            y = _rms(out.reshape(T, -1) * F.silu(g)) * w["norm"]
        elif mixer == "lightning":
            y = _rms(out.reshape(T, -1)) * w["norm"] * torch.sigmoid(g)
        else:
            y = (_rms(out) * w["norm"] if mixer == "decayed_linear_attention" else _rms(out)).reshape(T, -1) * F.silu(g)
    if mixer == "wkv":
        state = torch.cat((state, tail), -1)
    elif mixer == "state_space":
        state = torch.cat((tail, state), -1)
    return y @ w["o"].T, state


def _exact_logits(case, seed):
    width, _, heads, kv_heads, _ = SHAPES[case["shape"]]
    model = Model(_model_config(case).to_plan())                 # for the names and shapes of its tensors alone
    weights = _tensors({n: s for n, s in model.expected_tensors().items() if not s.ignored}, torch.bfloat16, seed)
    xs = [weights["model.embed_tokens.weight"][torch.tensor(p, device=DEV)].double() for p in _token_ids(case, seed)]
    for i in range(case["layers"]):
        w = {n[len(f"model.layers.{i}."):]: t.double() for n, t in weights.items() if n.startswith(f"model.layers.{i}.")}
        for r, x in enumerate(xs):
            h = _rms(x, w["input_layernorm.weight"])
            q, k, v = (h @ w[f"self_attn.{s}_proj.weight"].T + w[f"self_attn.{s}_proj.bias"] for s in "qkv")
            n = len(x)
            pos = torch.arange(n, device=DEV)
            a = _attend(_rotate(q.view(n, heads, 128), pos, THETA), _rotate(k.view(n, kv_heads, 128), pos, THETA),
                        v.view(n, kv_heads, 128), 0, 128 ** -0.5)
            x = x + a.reshape(n, -1) @ w["self_attn.o_proj.weight"].T
            h = _rms(x, w["post_attention_layernorm.weight"])
            xs[r] = x + (F.silu(h @ w["mlp.gate_proj.weight"].T) * (h @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T
    rows = _rms(torch.stack([x[-1] for x in xs]), weights["model.norm.weight"].double())
    return torch.cat([rows @ part.double().T for part in weights["lm_head.weight"].split(16384)], -1)
