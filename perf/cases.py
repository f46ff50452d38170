"""The work that a program on top of this engine has it do, as cases that can be timed and checked.

Seven kinds of case, each through an entry point that a program calls itself:

``step``       a decode step of a whole Qwen2-MoE model (``ModelRunner.step_ahead``, the call that the scheduler's executor
               makes for every token of a running batch): returns the logits of every request.
``decode``     attention of one new token per request over a long paged cache (``ops.functional.decode_attention``).
``attention``  a grouped-query attention layer over prompt portions: projections, rotation, cache write, attention, output.
``moe``        a sparse feed-forward: router, routed experts, gated shared expert.
``delta``      a gated delta rule layer (recurrent mixer with a matrix state per head) over prompts.
``memory``     a matrix-memory layer with exponential gates over prompts.
``latent``     an attention layer through a shared latent over prompt portions.

Layers are parts built from their description, as the engine builds them, and called with the step context that the
engine's runner hands them (pages in no order, requests of several lengths).  Sizes are those of ``bench.py``.
"""

import math
import random
import zlib

import torch

from mini_infer_b200.config import PartSpec, build_model_spec, part_class
from mini_infer_b200.engine.model import Model
from mini_infer_b200.engine.step import ModelRunner, StepEntry
from mini_infer_b200.ops import functional as F
from mini_infer_b200.ops.library import library
from mini_infer_b200.parts.base import (CacheBinding, KVGroupView, PagedCacheNeed, Runtime, StepContext,
                                        configure_matmul_exactness, precision_from_name)

PAGE = 16
DEVICE = "cuda:0"

# hidden size, heads, key/value heads, head size
ATTENTION = {"0.5b": (1024, 8, 2, 128), "a2.7b": (2048, 16, 16, 128), "57b-a14b": (3584, 28, 4, 128)}
# hidden size, experts, experts per token, expert width, shared expert's width
MOE = {"0.5b": (1024, 16, 2, 1024, 0), "a2.7b": (2048, 60, 4, 1408, 5632), "57b-a14b": (3584, 64, 8, 2560, 20480)}
# hidden size, heads, key heads, head size, value size
DELTA = {"0.5b": (1024, 8, 4, 128, 128), "a2.7b": (2048, 16, 8, 128, 128)}
# hidden size, heads, head size, value size
MEMORY = {"0.5b": (1024, 4, 128, 256), "2b": (2048, 4, 256, 512), "4b": (2560, 5, 256, 512)}
# hidden size, heads, unrotated and rotated size of a head, value size, latent size
LATENT = {"0.5b": (1024, 16, 64, 32, 64, 128), "2b": (2048, 16, 128, 64, 128, 512), "4b": (2560, 40, 64, 32, 64, 256)}
# layers, vocabulary of the whole models (attention and feed-forward as above)
STEP = {"0.5b": (6, 32000), "a2.7b": (4, 151936)}

THETA, EPS, TAPS, GATE_CAP = 1000000.0, 1e-6, 4, 15.0
YARN = {"theta": 10000.0, "factor": 16.0, "original": 4096, "fast": 32.0, "slow": 1.0}


def listed():
    return [
        # one user, a short conversation, a small model: latency and launches
        {"name": "step_small_1", "kind": "step", "size": "0.5b", "requests": 1, "context": 300},
        # the engine's headline: eight conversations of up to 2,048 tokens
        {"name": "step_8", "kind": "step", "size": "a2.7b", "requests": 8, "context": 2048},
        # a full server's decode attention, contexts of all lengths
        {"name": "decode_64", "kind": "decode", "size": "a2.7b", "requests": 64, "context": 3000, "window": 0},
        # one long prompt
        {"name": "attention_2048", "kind": "attention", "size": "a2.7b", "past": "0", "new": "2048", "window": 0,
         "dtype": "bfloat16"},
        # portions of several prompts in one step, behind what is cached of them already
        {"name": "attention_portions", "kind": "attention", "size": "57b-a14b", "past": "3000 0 517", "new": "777 250 101",
         "window": 0, "dtype": "bfloat16"},
        # the true 32-bit path: a portion of 512 tokens of a longer prompt
        {"name": "attention_f32", "kind": "attention", "size": "a2.7b", "past": "700", "new": "512", "window": 0,
         "dtype": "float32"},
        # the feed-forward of a decode step of many requests
        {"name": "moe_48", "kind": "moe", "size": "a2.7b", "tokens": 48, "dtype": "bfloat16"},
        # ... of a long prompt
        {"name": "moe_2048", "kind": "moe", "size": "a2.7b", "tokens": 2048, "dtype": "bfloat16"},
        # ... of a portion on the true 32-bit path
        {"name": "moe_f32", "kind": "moe", "size": "a2.7b", "tokens": 512, "dtype": "float32"},
        # two prompts through a recurrent mixer
        {"name": "delta_prompts", "kind": "delta", "size": "a2.7b", "new": "1501 547"},
        # one prompt through a matrix memory
        {"name": "memory_2048", "kind": "memory", "size": "2b", "new": "2048"},
        # one prompt's portion through latent attention
        {"name": "latent_portion", "kind": "latent", "size": "2b", "past": "1000", "new": "1024"},
    ]


def draw(rng):
    kind = rng.choice(["step", "decode", "attention", "attention", "moe", "moe", "delta", "memory", "latent"])
    if kind == "step":
        return {"kind": kind, "size": rng.choice(list(STEP)), "requests": rng.randint(1, 8), "context": _log(rng, 40, 2048)}
    if kind == "decode":
        return {"kind": kind, "size": rng.choice(list(ATTENTION)), "requests": _log(rng, 2, 64),
                "context": _log(rng, 200, 4000), "window": rng.choice([0, 0, 1024])}
    if kind == "attention":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        most = 2048 if dtype == "bfloat16" else 512
        past, new = _portions(rng, most, 3000 if dtype == "bfloat16" else 800)
        return {"kind": kind, "size": rng.choice(list(ATTENTION)[:2] if dtype == "float32" else list(ATTENTION)),
                "past": past, "new": new, "window": rng.choice([0, 0, 1024]), "dtype": dtype}
    if kind == "moe":
        dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
        size = rng.choice(list(MOE)[:2] if dtype == "float32" else list(MOE))
        return {"kind": kind, "size": size, "tokens": _log(rng, 1, 2048 if dtype == "bfloat16" else 512), "dtype": dtype}
    if kind == "latent":
        past, new = _portions(rng, 2048, 2000)
        return {"kind": kind, "size": rng.choice(list(LATENT)), "past": past, "new": new}
    return {"kind": kind, "size": rng.choice(list(DELTA if kind == "delta" else MEMORY)), "new": _portions(rng, 2048, 0)[1]}


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _portions(rng, most, past):
    """One to three requests that bring at most ``most`` tokens together, each behind up to ``past`` cached ones."""
    n = rng.randint(1, 3)
    new = [_log(rng, max(2, most // 32), most // n) for _ in range(n)]
    return (" ".join(str(rng.choice([0, rng.randint(0, past)])) for _ in new), " ".join(str(v) for v in new))


def _ints(text):
    return [int(v) for v in text.split()]


def _contexts(case):
    """Tokens of every request after this step: from a quarter of the longest up, in no order."""
    rng = random.Random(case["requests"] * 100003 + case["context"])
    lengths = [rng.randint(max(1, case["context"] // 4), case["context"]) for _ in range(case["requests"])]
    lengths[rng.randrange(len(lengths))] = case["context"]
    return lengths


# --------------------------------------------------------------------------- #
# weights
# --------------------------------------------------------------------------- #

class Weights:
    """Seeded normal tensors by name, in the manner of a checkpoint: ``declared`` are what a model or part asks for."""

    STD = {"conv": 0.3}

    def __init__(self, declared, seed, dtype):
        self._declared = {d.name: d for d in declared}
        self._seed, self._dtype = seed, dtype

    def names(self):
        return list(self._declared)

    def shape(self, name):
        return tuple(self._declared[name].shape)

    def dtype(self, name):
        return self._dtype

    def describe(self):
        return "seeded normal weights"

    def read(self, name):
        d = self._declared[name]
        w = _normal(tuple(d.shape), self._seed, name, self.STD.get(d.role, 0.02))
        return ((w + 1.0) if d.role == "norm" else w).to(self._dtype)

    __getitem__ = read

    def exact(self, name):
        return self.read(name).double()


def _normal(shape, seed, name, std=1.0):
    g = torch.Generator(device=DEVICE).manual_seed(zlib.crc32(f"{seed}:{name}".encode()))
    return torch.randn(shape, generator=g, device=DEVICE, dtype=torch.float32) * std


def _dtype(case):
    return torch.float32 if case.get("dtype") == "float32" else torch.bfloat16


def _runtime(case):
    library()
    configure_matmul_exactness()
    return Runtime(precision_from_name(case.get("dtype", "bfloat16")), torch.device(DEVICE))


# --------------------------------------------------------------------------- #
# what a program has before the call
# --------------------------------------------------------------------------- #

def _part(case):
    """The layer's part, not loaded."""
    kind, size = case["kind"], case["size"]
    if kind == "attention":
        H, nh, nkv, d = ATTENTION[size]
        return part_class("mixer", "gqa_attention")({
            "hidden_size": H, "num_heads": nh, "num_kv_heads": nkv, "head_dim": d, "bias": True, "window": case["window"],
            "position": PartSpec("rope", {"head_dim": d, "theta": THETA})}, "")
    if kind == "moe":
        H, E, K, mI, sI = MOE[size]
        return part_class("feed_forward", "sparse_moe")({
            "hidden_size": H, "num_experts": E, "top_k": K, "expert_intermediate_size": mI,
            "shared_intermediate_size": sI, "norm_topk_prob": False}, "")
    if kind == "delta":
        H, nh, nkv, d, dv = DELTA[size]
        return part_class("mixer", "gated_delta")({
            "hidden_size": H, "num_heads": nh, "num_kv_heads": nkv, "head_dim": d, "value_dim": dv, "conv": TAPS,
            "eps": EPS}, "")
    if kind == "memory":
        H, nh, d, dv = MEMORY[size]
        return part_class("mixer", "matrix_lstm")({
            "hidden_size": H, "num_heads": nh, "head_dim": d, "value_dim": dv, "gate_cap": GATE_CAP, "eps": EPS}, "")
    H, nh, d, r, e, c = LATENT[size]
    return part_class("mixer", "latent_attention")({
        "hidden_size": H, "num_heads": nh, "head_dim": d, "rot_dim": r, "value_dim": e, "kv_rank": c, "q_rank": 0,
        "window": 0, "scale": (d + r) ** -0.5, "eps": EPS, "output_gate": True,
        "position": PartSpec("rope_yarn", dict(YARN, head_dim=r, pairing="neighbours"))}, "")


def _lengths(case):
    """Cached and new tokens of every request."""
    if "requests" in case:
        return [n - 1 for n in _contexts(case)], [1] * case["requests"]
    new = _ints(case["new"]) if "new" in case else [case["tokens"]]
    return _ints(case["past"]) if "past" in case else [0] * len(new), new


def _pages(lengths, seed):
    """A page table per request, of pages in no order: ``[requests, most pages]``, -1 where there is none."""
    counts = [-(-n // PAGE) for n in lengths]
    order = list(range(sum(counts)))
    random.Random(seed).shuffle(order)
    table = torch.full((len(lengths), max(counts)), -1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(counts):
        table[b, :n] = torch.tensor(order[at:at + n], dtype=torch.int32)
        at += n
    return table, len(order)


def _context(part, case, seed):
    """The step context of a layer: requests with ``past`` cached tokens that bring ``new`` ones, and the layer's cache."""
    past, new = _lengths(case)
    need = None if case["kind"] == "moe" else part.cache_need()
    B, T = len(new), sum(new)
    ends = [p + n for p, n in zip(past, new)]
    table, pages = _pages(ends, seed)
    req = torch.repeat_interleave(torch.arange(B), torch.tensor(new))
    pos = torch.cat([torch.arange(p, e) for p, e in zip(past, ends)])
    starts = [sum(new[:b]) for b in range(B + 1)]
    dev = lambda t: torch.as_tensor(t, dtype=torch.int32).to(DEVICE)
    groups, states = [], []
    if isinstance(need, PagedCacheNeed):
        tensors = {name: _normal((1, pages) + tuple(shape), seed, "cache " + name).to(dtype or _dtype(case))
                   for name, shape, dtype in need.tensors(PAGE)}
        groups.append(KVGroupView(dev(table), dev(table[req, pos // PAGE] * PAGE + pos % PAGE), PAGE, tensors))
    elif need is not None:
        states.append(torch.zeros((B + 1,) + tuple(need.shape), dtype=need.dtype or torch.float32, device=DEVICE))
    leading = next((b for b, n in enumerate(new) if n != 1), B)
    return StepContext(
        num_tokens=T, num_requests=B, max_q_len=max(new), max_kv_len=max(ends), all_decode=max(new) == 1,
        token_ids=dev([0] * T), positions=dev(pos), q_start=dev(starts), kv_len=dev(ends), req_of_token=dev(req),
        state_slot=dev(list(range(B))), fresh=dev([int(p == 0) for p in past]), kv_groups=groups, states=states,
        scratch={}, num_leading_decodes=leading, leading_decodes_max_kv_len=max(ends[:leading], default=0),
        host_q_start=starts, host_kv_len=ends, host_state_slot=list(range(B)))


def _prepare_step(case, seed):
    rt = _runtime(case)
    config = _step_config(case)
    model = Model(build_model_spec(config))
    model.load(Weights(model.tensor_decls(), seed, torch.bfloat16), rt)
    lengths = _contexts(case)
    runner = ModelRunner(model, rt, page_size=PAGE, num_pages=sum(-(-n // PAGE) + 1 for n in lengths),
                         max_requests=len(lengths), max_tokens_per_step=max(lengths + [len(lengths)]),
                         max_context=max(lengths) + 1)
    tokens = _step_tokens(case, seed)
    for b, row in enumerate(tokens):
        runner.add_request(b)
        if len(row) > 1:
            runner.step([StepEntry(b, row[:-1])])
    last = torch.tensor([row[-1] for row in tokens], dtype=torch.int32, device=DEVICE)
    state = {"runner": runner, "requests": list(range(len(lengths))), "tokens": last}
    _run_step(state)            # a serving process captures its decode steps before the first request
    return state


def _step_config(case):
    H, nh, nkv, d = ATTENTION[case["size"]]
    _, E, K, mI, sI = MOE[case["size"]]
    layers, vocab = STEP[case["size"]]
    return {"architectures": ["Qwen2MoeForCausalLM"], "model_type": "qwen2_moe", "vocab_size": vocab, "hidden_size": H,
            "intermediate_size": 4 * mI, "num_hidden_layers": layers, "num_attention_heads": nh, "head_dim": d,
            "num_key_value_heads": nkv, "rms_norm_eps": EPS, "rope_theta": THETA, "max_position_embeddings": 8192,
            "tie_word_embeddings": False, "hidden_act": "silu", "num_experts": E, "num_experts_per_tok": K,
            "moe_intermediate_size": mI, "shared_expert_intermediate_size": sI, "norm_topk_prob": False,
            "decoder_sparse_step": 1, "mlp_only_layers": [], "use_sliding_window": False}


def _step_tokens(case, seed):
    rng = random.Random(seed)
    vocab = STEP[case["size"]][1]
    return [[rng.randrange(vocab) for _ in range(n)] for n in _contexts(case)]


def _prepare_decode(case, seed):
    library()
    _, nh, nkv, d = ATTENTION[case["size"]]
    lengths = _contexts(case)
    B = len(lengths)
    table, pages = _pages(lengths, seed)
    split = F.decode_split_size()
    splits = -(-max(lengths) // split)
    return {"q": _normal((B, nh, d), seed, "q").bfloat16(),
            "k": _normal((pages, nkv, PAGE, d), seed, "k").bfloat16(), "v": _normal((pages, nkv, PAGE, d), seed, "v").bfloat16(),
            "table": table.to(DEVICE), "starts": torch.arange(B + 1, dtype=torch.int32, device=DEVICE),
            "lengths": torch.tensor(lengths, dtype=torch.int32, device=DEVICE), "splits": splits, "split": split,
            "part_o": torch.empty(B * nh * splits * d, dtype=torch.float32, device=DEVICE),
            "part_ml": torch.empty(B * nh * splits * 2, dtype=torch.float32, device=DEVICE), "window": case["window"]}


def prepare(case, seed):
    if case["kind"] == "step":
        return dict(_prepare_step(case, seed), kind="step")
    if case["kind"] == "decode":
        return dict(_prepare_decode(case, seed), kind="decode")
    part = _part(case)
    part.load(Weights(part.tensor_decls(), seed, _dtype(case)), _runtime(case))
    context = _context(part, case, seed)
    return {"kind": case["kind"], "part": part, "x": _input(case, seed), "context": context,
            "binding": CacheBinding("state" if context.states else "kv", 0, 0, True)}


def _input(case, seed):
    """What a norm hands a layer: rows of unit root mean square."""
    T = sum(_lengths(case)[1])
    table = {"moe": MOE, "attention": ATTENTION, "delta": DELTA, "memory": MEMORY, "latent": LATENT}[case["kind"]]
    x = _normal((T, table[case["size"]][0]), seed, "x")
    return (x / x.pow(2).mean(-1, keepdim=True).sqrt()).to(_dtype(case))


# --------------------------------------------------------------------------- #
# the call
# --------------------------------------------------------------------------- #

def _run_step(s):
    logits = s["runner"].step_ahead(s["requests"], s["tokens"])
    s["runner"].drop_ahead(s["requests"])       # the next pass decodes the same tokens again
    return logits


@torch.no_grad()
def run(state):
    kind = state["kind"]
    if kind == "step":
        return _run_step(state)
    if kind == "decode":
        s = state
        return F.decode_attention(s["q"], s["k"], s["v"], s["table"], s["starts"], s["lengths"], s["part_o"], s["part_ml"],
                                  s["splits"], s["window"], split=s["split"])
    part, x, ctx = state["part"], state["x"], state["context"]
    if kind == "moe":
        return part.forward(x, ctx)
    if ctx.states:
        ctx.states[0].zero_()                   # a request's state when it is admitted
        return part.forward(x, ctx, state["binding"]), ctx.states[0]
    y = part.forward(x, ctx, state["binding"])
    return (y,) + tuple(ctx.kv_groups[0].tensors.values())


# --------------------------------------------------------------------------- #
# what a pass cannot do without
# --------------------------------------------------------------------------- #

def _pairs(past, new, window):
    total = 0
    for p, n in zip(past, new):
        full = n * p + n * (n + 1) // 2
        over = max(0, p + n - window) if window else 0      # positions with more than `window` keys up to them
        cut = min(over, n)
        total += full - sum(range(over - cut + 1, over + 1))
    return total


def _moe_work(size, T, item):
    H, E, K, mI, sI = MOE[size]
    used = E * (1.0 - (1.0 - K / E) ** T)
    return (item * (used * 3 * mI * H + 3 * sI * H + (E + 1) * H + T * H) + 4 * T * H,
            2.0 * T * H * (3 * K * mI + 3 * sI + E + 1))


def _attention_work(size, past, new, window, item):
    H, nh, nkv, d = ATTENTION[size]
    T = sum(new)
    keys = sum(n + min(p, window) if window else n + p for p, n in zip(past, new))
    weights = (nh + 2 * nkv) * d * H + nh * d * H
    return (item * (weights + T * H + 2 * (keys + T) * nkv * d) + 4 * T * H,
            2.0 * T * weights + 4.0 * d * nh * _pairs(past, new, window))


def work(case):
    item = 4 if case.get("dtype") == "float32" else 2
    kind, size = case["kind"], case["size"]
    if kind == "moe":
        by, fl = _moe_work(size, case["tokens"], item)
        return {"bytes": by, "flops": fl}
    past, new = _lengths(case)
    T = sum(new)
    if kind == "step":
        layers, vocab = STEP[size]
        H = MOE[size][0]
        a, m = _attention_work(size, past, new, 0, item), _moe_work(size, T, item)
        return {"bytes": layers * (a[0] + m[0]) + item * vocab * H + 4 * T * vocab, "flops": layers * (a[1] + m[1]) + 2.0 * T * vocab * H}
    if kind == "attention":
        by, fl = _attention_work(size, past, new, case["window"], item)
        return {"bytes": by, "flops": fl}
    if kind == "decode":
        _, nh, nkv, d = ATTENTION[size]
        keys = sum(min(p + 1, case["window"]) if case["window"] else p + 1 for p in past)
        return {"bytes": item * (2 * keys * nkv * d + 2 * T * nh * d), "flops": 4.0 * keys * nh * d}
    if kind == "latent":
        H, nh, d, r, e, c = LATENT[size]
        weights = H * (nh * (d + r) + c + r + 2 * nh * e)
        keys = sum(past) + T
        return {"bytes": item * (weights + nh * (d + e) * c + T * H + (keys + T) * (c + r)) + 4 * T * H,
                "flops": 2.0 * T * weights + 2.0 * keys * nh * (d + e) * c + 2.0 * _pairs(past, new, 0) * nh * (d + r + e)}
    if kind == "delta":
        H, nh, nkv, d, dv = DELTA[size]
        weights = H * (2 * nkv * d + 3 * nh * dv + 2 * nh)
        state = len(new) * nh * d * dv
        return {"bytes": item * (weights + T * H) + 4 * T * H + 8 * state, "flops": 2.0 * T * weights + 6.0 * T * nh * d * dv}
    H, nh, d, dv = MEMORY[size]
    weights = H * (2 * nh * d + 3 * nh * dv + 2 * nh)
    state = len(new) * nh * d * dv
    return {"bytes": item * (weights + T * H) + 4 * T * H + 8 * state, "flops": 2.0 * T * weights + 4.0 * T * nh * d * dv}


# Relative errors of another correct implementation: about four times the distance that the path shows from `exact`.
def tolerance(case):
    if case.get("dtype") == "float32":
        return {"rel": 2.5e-5 if case["kind"] == "attention" else 8e-6}     # angles of long positions in 32 bits
    return {"rel": {"step": 5e-2, "decode": 7e-3, "attention": 1.5e-2, "moe": 1.2e-2, "delta": 7e-3, "memory": 2e-2,
                    "latent": 1.5e-2}[case["kind"]]}


# --------------------------------------------------------------------------- #
# the same in 64 bits
# --------------------------------------------------------------------------- #

def _rms(x, eps=EPS):
    return x / (x.pow(2).mean(-1, keepdim=True) + eps).sqrt()


def _silu(x):
    return x * torch.sigmoid(x)


def _softmax_attention(q, k, v, first, scale, window=0):
    """``q [n, H, d]`` at positions ``first ...`` over keys ``k [S, H, d]``, values ``v [S, H, e]``: ``[n, H, e]``."""
    at = torch.arange(first, first + q.shape[0], device=q.device)[:, None]
    key = torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = (key > at) | ((key <= at - window) if window else torch.zeros((), dtype=torch.bool, device=q.device))
    out = [torch.softmax(((q[:, h] @ k[:, h].T) * scale).masked_fill(hidden, -math.inf), -1) @ v[:, h]
           for h in range(q.shape[1])]
    return torch.stack(out, 1)


def _rotate(x, positions, freqs, neighbours=False, magnitude=1.0):
    """``x [n, heads, r]`` turned by position, pairs of halves or of neighbours."""
    a = positions.double()[:, None] * freqs[None, :]
    cos, sin = torch.cos(a)[:, None, :] * magnitude, torch.sin(a)[:, None, :] * magnitude
    half = x.shape[-1] // 2
    u, w = (x[..., 0::2], x[..., 1::2]) if neighbours else (x[..., :half], x[..., half:])
    a, b = u * cos - w * sin, w * cos + u * sin
    return torch.stack([a, b], -1).flatten(-2) if neighbours else torch.cat([a, b], -1)


def _frequencies(r, theta):
    return theta ** (-2.0 * torch.arange(r // 2, dtype=torch.float64, device=DEVICE) / r)


def _exact_gqa(x, W, prefix, size, past, new, window, cached):
    """One attention layer in 64 bits: ``cached(b) -> (keys, values)`` of request ``b``'s earlier tokens.  Returns the
    output and every request's new keys and values."""
    H, nh, nkv, d = ATTENTION[size]
    q, k, v = (x @ W.exact(f"{prefix}{n}_proj.weight").T + W.exact(f"{prefix}{n}_proj.bias") for n in "qkv")
    freqs = _frequencies(d, THETA)
    out, rows, at = [], [], 0
    for b, (p, n) in enumerate(zip(past, new)):
        pos = torch.arange(p, p + n, device=DEVICE)
        qb = _rotate(q[at:at + n].view(n, nh, d), pos, freqs)
        kb = _rotate(k[at:at + n].view(n, nkv, d), pos, freqs)
        vb = v[at:at + n].view(n, nkv, d)
        rows.append((kb, vb))
        ck, cv = cached(b)
        kk, vv = torch.cat([ck, kb]), torch.cat([cv, vb])
        rep = nh // nkv
        out.append(_softmax_attention(qb, kk.repeat_interleave(rep, 1), vv.repeat_interleave(rep, 1), p, d ** -0.5,
                                      window).reshape(n, nh * d))
        at += n
    return torch.cat(out) @ W.exact(prefix + "o_proj.weight").T, rows


def _paged(cache, table, b, n):
    """The first ``n`` rows of request ``b`` out of pages ``[pages, heads, page, size]``: ``[n, heads, size]``."""
    pages = table[b, :-(-n // PAGE)].long().to(cache.device)
    return cache[pages].transpose(1, 2).reshape(-1, cache.shape[1], cache.shape[3])[:n].double()


def _stored(cache, table, past, rows):
    """The pages after ``rows[b] [n, heads, size]`` have been written behind ``past[b]`` tokens."""
    out = cache.double()
    for b, (p, r) in enumerate(zip(past, rows)):
        pos = torch.arange(p, p + r.shape[0])
        out[table[b, pos // PAGE].long().to(out.device), :, (pos % PAGE).to(out.device)] = r
    return out


def _exact_moe(x, W, prefix, size):
    H, E, K, mI, sI = MOE[size]
    glu = lambda h, p: (_silu(h @ W.exact(p + "gate_proj.weight").T) * (h @ W.exact(p + "up_proj.weight").T)) \
        @ W.exact(p + "down_proj.weight").T
    weight, chosen = torch.softmax(x @ W.exact(prefix + "gate.weight").T, -1).topk(K, -1)
    y = torch.zeros_like(x)
    for e in range(E):
        token, slot = (chosen == e).nonzero(as_tuple=True)
        if token.numel():
            y.index_add_(0, token, glu(x[token], f"{prefix}experts.{e}.") * weight[token, slot][:, None])
    if sI:
        y = y + torch.sigmoid(x @ W.exact(prefix + "shared_expert_gate.weight").T) * glu(x, prefix + "shared_expert.")
    return y


def _exact_step(case, seed):
    layers, _ = STEP[case["size"]]
    _, _, nkv, d = ATTENTION[case["size"]]
    W = Weights(Model(build_model_spec(_step_config(case))).tensor_decls(), seed, torch.bfloat16)
    tokens = _step_tokens(case, seed)
    new = [len(t) for t in tokens]
    past = [0] * len(new)
    none = torch.empty(0, nkv, d, dtype=torch.float64, device=DEVICE)
    h = W.exact("model.embed_tokens.weight")[torch.tensor([t for row in tokens for t in row], device=DEVICE)]
    for i in range(layers):
        p = f"model.layers.{i}."
        y, _ = _exact_gqa(_rms(h) * W.exact(p + "input_layernorm.weight"), W, p + "self_attn.", case["size"], past, new, 0,
                          lambda b: (none, none))
        h = h + y
        h = h + _exact_moe(_rms(h) * W.exact(p + "post_attention_layernorm.weight"), W, p + "mlp.", case["size"])
    ends = torch.tensor(new, device=DEVICE).cumsum(0) - 1
    return (_rms(h[ends]) * W.exact("model.norm.weight")) @ W.exact("lm_head.weight").T


def _exact_decode(case, seed):
    _, nh, nkv, d = ATTENTION[case["size"]]
    s = _prepare_decode(case, seed)
    out, rep = [], nh // nkv
    for b, n in enumerate(_contexts(case)):
        k, v = (_paged(s[t], s["table"], b, n).repeat_interleave(rep, 1) for t in ("k", "v"))
        out.append(_softmax_attention(s["q"][b:b + 1].double(), k, v, n - 1, d ** -0.5, case["window"]))
    return torch.cat(out)


def _exact_delta(x, W, case):
    H, nh, nkv, d, dv = DELTA[case["size"]]
    out, at = [], 0
    for n in _ints(case["new"]):
        h = x[at:at + n]
        at += n

        def conv(name):
            w = W.exact(name + ".conv")
            p = torch.cat([torch.zeros(TAPS - 1, w.shape[0], dtype=torch.float64, device=DEVICE), h @ W.exact(name).T])
            return _silu(sum(p[j:j + n] * w[:, j] for j in range(TAPS)))
        unit = lambda t: t / (t.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
        q = (unit(conv("q").view(n, nkv, d)) * d ** -0.5).repeat_interleave(nh // nkv, 1)
        k = unit(conv("k").view(n, nkv, d)).repeat_interleave(nh // nkv, 1)
        v = conv("v").view(n, nh, dv)
        beta = torch.sigmoid(h @ W.exact("b").T)
        g = torch.exp(-torch.exp(W.exact("A_log")) * torch.nn.functional.softplus(h @ W.exact("a").T + W.exact("dt_bias")))
        S = torch.zeros(nh, d, dv, dtype=torch.float64, device=DEVICE)
        o = torch.empty(n, nh, dv, dtype=torch.float64, device=DEVICE)
        for t in range(n):
            S = S * g[t, :, None, None]
            u = beta[t, :, None] * (v[t] - torch.bmm(k[t, :, None, :], S)[:, 0])
            S = S + k[t, :, :, None] * u[:, None, :]
            o[t] = torch.bmm(q[t, :, None, :], S)[:, 0]
        y = (_rms(o) * W.exact("norm")).reshape(n, nh * dv) * _silu(h @ W.exact("g").T)
        out.append(y @ W.exact("o").T)
    return torch.cat(out)


def _exact_memory(x, W, case):
    """The whole history weighed at once: a write at ``j`` counts ``exp(i_j + sum of f after j)`` at ``t``."""
    H, nh, d, dv = MEMORY[case["size"]]
    cap = lambda z: GATE_CAP * torch.tanh(z / GATE_CAP)
    out, at = [], 0
    for n in _ints(case["new"]):
        h = x[at:at + n]
        at += n
        q, k = (h @ W.exact("q").T).view(n, nh, d) * d ** -0.5, (h @ W.exact("k").T).view(n, nh, d)
        v = (h @ W.exact("v").T).view(n, nh, dv)
        i = cap(h @ W.exact("i").T + W.exact("i.b"))
        f = torch.nn.functional.logsigmoid(cap(h @ W.exact("f").T + W.exact("f.b"))).cumsum(0)
        later = torch.ones(n, n, dtype=torch.bool, device=DEVICE).triu(1)
        o = torch.empty(n, nh, dv, dtype=torch.float64, device=DEVICE)
        for a in range(nh):
            w = (f[:, None, a] - f[None, :, a] + i[None, :, a]).masked_fill(later, -math.inf)
            m = torch.maximum(w.max(1).values, f[:, a])         # the running maximum starts at 0
            s = torch.exp(w - m[:, None]) * (q[:, a] @ k[:, a].T)
            o[:, a] = (s @ v[:, a]) / (torch.maximum(s.sum(1).abs(), torch.exp(-m)) + 1e-6)[:, None]
        y = _rms(o).reshape(n, nh * dv) * W.exact("norm") * torch.sigmoid(h @ W.exact("g").T)
        out.append(y @ W.exact("o").T)
    return torch.cat(out)


def _yarn(r):
    """YaRN: pairs that turn fast over the original context keep their frequency, slow ones are stretched, a ramp between."""
    at = lambda turns: r * math.log(YARN["original"] / (turns * 2 * math.pi)) / (2 * math.log(YARN["theta"]))
    low, high = max(math.floor(at(YARN["fast"])), 0), min(math.ceil(at(YARN["slow"])), r - 1)
    ramp = ((torch.arange(r // 2, dtype=torch.float64, device=DEVICE) - low) / max(high - low, 1e-3)).clamp(0, 1)
    f = _frequencies(r, YARN["theta"])
    return f * (1 - ramp) + f / YARN["factor"] * ramp, 0.1 * math.log(YARN["factor"]) + 1.0


def _exact_latent(x, W, case, cache, table):
    H, nh, d, r, e, c = LATENT[case["size"]]
    past, new = _lengths(case)
    freqs, magnitude = _yarn(r)
    q, z = (x @ W.exact("q").T).view(-1, nh, d + r), x @ W.exact("dkv").T
    uk, uv = W.exact("uk").view(nh, d, c), W.exact("uv").view(nh, e, c)
    out, rows, at = [], [], 0
    for b, (p, n) in enumerate(zip(past, new)):
        pos = torch.arange(p, p + n, device=DEVICE)
        qb, zb = q[at:at + n], z[at:at + n]
        at += n
        qb = torch.cat([qb[..., :d], _rotate(qb[..., d:], pos, freqs, True, magnitude)], -1)
        row = torch.cat([_rms(zb[:, :c]) * W.exact("dkv.norm"), _rotate(zb[:, None, c:], pos, freqs, True, magnitude)[:, 0]], -1)
        rows.append(row[:, None])
        kv = torch.cat([_paged(cache, table, b, p)[:, 0], row])
        k = torch.cat([torch.einsum("sc,hdc->shd", kv[:, :c], uk), kv[:, None, c:].expand(-1, nh, -1)], -1)
        v = torch.einsum("sc,hec->she", kv[:, :c], uv)
        out.append(_softmax_attention(qb, k, v, p, (d + r) ** -0.5).reshape(n, nh * e))
    y = torch.cat(out) * torch.sigmoid(x @ W.exact("g").T)
    return y @ W.exact("o").T, rows


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "decode":
        return _exact_decode(case, seed)
    part = _part(case)
    W = Weights(part.tensor_decls(), seed, _dtype(case))
    x = _input(case, seed).double()
    if kind == "moe":
        return _exact_moe(x, W, "", case["size"])
    if kind == "delta":
        return _exact_delta(x, W, case), None
    if kind == "memory":
        return _exact_memory(x, W, case), None
    past, new = _lengths(case)
    view = _context(part, case, seed).kv_groups[0]
    table = view.block_table.cpu()
    if kind == "latent":
        cache = view.tensors["latent"][0]
        y, rows = _exact_latent(x, W, case, cache, table)
        return y, _stored(cache, table, past, rows)[None]
    k, v = view.tensors["k"][0], view.tensors["v"][0]
    y, rows = _exact_gqa(x, W, "", case["size"], past, new, case["window"],
                         lambda b: (_paged(k, table, b, past[b]), _paged(v, table, b, past[b])))
    return y, _stored(k, table, past, [r[0] for r in rows])[None], _stored(v, table, past, [r[1] for r in rows])[None]
