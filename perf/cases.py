"""What this library is timed at: the work that its users have it do, over the real range of sizes.

Twelve listed cases and ``draw``, which gives more of the same ranges.  Whole calls go through ``Engine.step`` (what the
Python entry point, the command line and ``bin/trace_run`` call); single layers go through the parts that a model is put
together from, with the paged cache they run on.  Sizes are those of the benchmark's and the tests' configurations.
"""

from __future__ import annotations

import math
import random

import torch

from gtar_kimik3_public_b200.engine.engine import Engine, StepEntry
from gtar_kimik3_public_b200.engine.step import SequenceStep, plan_step
from gtar_kimik3_public_b200.models.model import Model
from gtar_kimik3_public_b200.ops.functional import DecodeWork, PagedKV
from gtar_kimik3_public_b200.parts.base import build_part
from gtar_kimik3_public_b200.registry import architecture, config_from_dict
from gtar_kimik3_public_b200.sampling.sampler import SamplingParams, choose

DEVICE = torch.device("cuda:0")
PAGE = 64
EPS = 1e-6
ROPE_BASE = 1e6

_COMMON = {"arch": "transformer", "head_dim": 128, "rms_norm_eps": 1e-6, "rope_theta": 1e6, "initializer_range": 0.02}
MODELS = {
    # 3 layers whose widths are no powers of two: the 32-bit check configuration
    "tiny": {"arch": "transformer", "vocab_size": 384, "hidden_size": 80, "intermediate_size": 224, "num_hidden_layers": 3,
             "num_attention_heads": 6, "num_key_value_heads": 2, "head_dim": 32, "rms_norm_eps": 1e-5, "rope_theta": 1e6,
             "tie_word_embeddings": False, "initializer_range": 0.02, "max_position_embeddings": 256},
    # two layers of the benchmark model's sizes with a small vocabulary: the 32-bit check path at real layer sizes
    "layers_06b": {**_COMMON, "vocab_size": 3000, "hidden_size": 1024, "intermediate_size": 3072, "num_hidden_layers": 2,
                   "num_attention_heads": 16, "num_key_value_heads": 8, "tie_word_embeddings": True, "max_position_embeddings": 2048},
    # the benchmark model, whole
    "qwen3_06b": {**_COMMON, "vocab_size": 151936, "hidden_size": 1024, "intermediate_size": 3072, "num_hidden_layers": 28,
                  "num_attention_heads": 16, "num_key_value_heads": 8, "tie_word_embeddings": True, "max_position_embeddings": 4096},
}
# (hidden, query heads, kv heads, feed-forward) of the three benchmark configurations; heads of 128
LAYERS = {"0.6b": (1024, 16, 8, 3072), "4b": (2560, 32, 8, 9728), "8b": (4096, 32, 8, 12288)}
HEAD = 128


def listed():
    return [
        # one person's short question to the whole benchmark model: a prompt, then tokens one at a time at batch 1
        {"name": "chat_one", "kind": "engine", "model": "qwen3_06b", "dtype": "bfloat16", "prompts": "33", "steps": 8},
        # the 32-bit check of a tiny model, whole prompts and single tokens of an unequal batch: launches and latency
        {"name": "check_tiny", "kind": "engine", "model": "tiny", "dtype": "float32", "prompts": "1,9,40,64", "steps": 24},
        # the 32-bit check at real layer sizes: prompts of a few hundred tokens, then single tokens after them
        {"name": "check_layers", "kind": "engine", "model": "layers_06b", "dtype": "float32", "prompts": "37,256,512", "steps": 8},
        # an attention layer in a decode step of eight requests of unequal lengths
        {"name": "attention_decode_8", "kind": "attention", "layer": "4b", "new": "1,1,1,1,1,1,1,1",
         "past": "255,700,1201,1777,2303,2900,3517,4095"},
        # an attention layer over the benchmark's prompt of 2,048 tokens
        {"name": "attention_prompt", "kind": "attention", "layer": "0.6b", "new": "2048", "past": "0"},
        # an attention layer over eight unequal prompts that start together
        {"name": "attention_prompts_8", "kind": "attention", "layer": "4b", "new": "256,701,1202,1778,2304,2901,3518,4096",
         "past": "0,0,0,0,0,0,0,0"},
        # a feed-forward in a decode step of eight, and of 64 requests
        {"name": "mlp_decode_8", "kind": "mlp", "layer": "4b", "tokens": 8},
        {"name": "mlp_decode_64", "kind": "mlp", "layer": "8b", "tokens": 64},
        # a feed-forward over the benchmark's prompt
        {"name": "mlp_prompt", "kind": "mlp", "layer": "0.6b", "tokens": 2048},
        # the token choice of 64 requests with temperature and top-k
        {"name": "sample_64", "kind": "sample", "rows": 64, "vocab": 151936, "temperature": 0.8, "top_k": 50},
        # a recurrent layer (delta rule with a decay per key channel) over a prompt of 2,048 tokens
        {"name": "delta_prompt", "kind": "delta", "hidden": 1024, "heads": 8, "new": "2048"},
        # routed experts in a decode step of eight requests
        {"name": "experts_decode_8", "kind": "experts", "hidden": 2048, "ff": 1024, "experts": 64, "top": 6, "groups": 8, "keep": 4,
         "tokens": 8},
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _join(numbers):
    return ",".join(str(n) for n in numbers)


def draw(rng: random.Random):
    kind = rng.choice(["chat", "check", "check_layers", "decode", "decode", "prompt", "prompts", "mlp", "mlp", "mlp", "sample", "delta", "experts"])
    if kind == "chat":
        n = rng.randint(1, 4)
        return {"kind": "engine", "model": "qwen3_06b", "dtype": "bfloat16", "prompts": _join(_log_int(rng, 3, 64) for _ in range(n)),
                "steps": rng.randint(3, 6)}
    if kind == "check":
        return {"kind": "engine", "model": "tiny", "dtype": "float32", "prompts": _join(rng.randint(1, 64) for _ in range(rng.randint(1, 6))),
                "steps": rng.randint(8, 24)}
    if kind == "check_layers":
        return {"kind": "engine", "model": "layers_06b", "dtype": "float32",
                "prompts": _join(_log_int(rng, 5, 384) for _ in range(rng.randint(1, 3))), "steps": rng.randint(3, 8)}
    layer = rng.choice(["0.6b", "4b", "8b"])
    if kind == "decode":
        n = _log_int(rng, 1, 64)
        return {"kind": "attention", "layer": layer, "new": _join([1] * n), "past": _join(_log_int(rng, 64, 4095) for _ in range(n))}
    if kind == "prompt":
        return {"kind": "attention", "layer": layer, "new": str(_log_int(rng, 65, 4096)), "past": "0"}
    if kind == "prompts":  # unequal prompts, some of them continuing a conversation
        n = rng.randint(2, 6)
        return {"kind": "attention", "layer": rng.choice(["0.6b", "4b"]), "new": _join(_log_int(rng, 32, 2500) for _ in range(n)),
                "past": _join(rng.choice([0, 0, rng.randint(1, 1500)]) for _ in range(n))}
    if kind == "mlp":
        return {"kind": "mlp", "layer": layer, "tokens": rng.choice([_log_int(rng, 1, 64), _log_int(rng, 1, 64), _log_int(rng, 65, 4096)])}
    if kind == "sample":
        return {"kind": "sample", "rows": _log_int(rng, 1, 64), "vocab": rng.randint(32000, 152064),
                "temperature": rng.choice([0.0, 0.6, 0.8, 1.0]), "top_k": rng.choice([0, 1, 20, 50, 200])}
    if kind == "delta":
        width = rng.choice([1024, 2048])
        return {"kind": "delta", "hidden": width, "heads": width // 128, "new": _join(_log_int(rng, 33, 1024) for _ in range(rng.randint(1, 3)))}
    if rng.random() < 0.5:
        return {"kind": "experts", "hidden": 1024, "ff": 768, "experts": 32, "top": 4, "groups": 4, "keep": 2, "tokens": _log_int(rng, 1, 2048)}
    return {"kind": "experts", "hidden": 2048, "ff": 1024, "experts": 64, "top": 6, "groups": 8, "keep": 4, "tokens": _log_int(rng, 1, 2048)}


# ------------------------------------------------------------------ inputs, from the seed alone
class _Draws:
    """Values in the order they are asked for: matrices N(0, 0.02), norm weights about one, activations of unit size."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def normal(self, *shape, mean=0.0, std=1.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.gen, device=DEVICE) * std + mean).to(dtype)

    def matrix(self, *shape, std=0.02):
        return self.normal(*shape, std=std, dtype=torch.bfloat16)

    def vector(self, n):
        return self.normal(n, mean=1.0, std=0.1)

    def ints(self, high, *shape):
        return torch.randint(0, high, shape, generator=self.gen, device=DEVICE, dtype=torch.int32)


def _numbers(text):
    return [int(n) for n in str(text).split(",")]


def _engine_inputs(case, seed):
    cfg = MODELS[case["model"]]
    d = _Draws(seed)
    h, ff, dim = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    nq, nkv, vocab = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["vocab_size"]
    t = {"model.embed_tokens.weight": d.matrix(vocab, h)}
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        t[p + "input_layernorm.weight"], t[p + "post_attention_layernorm.weight"] = d.vector(h), d.vector(h)
        t[p + "self_attn.q_proj.weight"], t[p + "self_attn.k_proj.weight"] = d.matrix(nq * dim, h), d.matrix(nkv * dim, h)
        t[p + "self_attn.v_proj.weight"], t[p + "self_attn.o_proj.weight"] = d.matrix(nkv * dim, h), d.matrix(h, nq * dim)
        t[p + "self_attn.q_norm.weight"], t[p + "self_attn.k_norm.weight"] = d.vector(dim), d.vector(dim)
        t[p + "mlp.gate_proj.weight"], t[p + "mlp.up_proj.weight"], t[p + "mlp.down_proj.weight"] = d.matrix(ff, h), d.matrix(ff, h), d.matrix(h, ff)
    t["model.norm.weight"] = d.vector(h)
    if not cfg["tie_word_embeddings"]:
        t["lm_head.weight"] = d.matrix(vocab, h)
    prompts = _numbers(case["prompts"])
    ids = d.ints(vocab, len(prompts), max(prompts) + case["steps"]).tolist()
    return cfg, t, [row[:n + case["steps"]] for row, n in zip(ids, prompts)], prompts


def _attention_inputs(case, seed):
    hidden, nq, nkv, _ = LAYERS[case["layer"]]
    d = _Draws(seed)
    tensors = {"q_proj.weight": d.matrix(nq * HEAD, hidden), "k_proj.weight": d.matrix(nkv * HEAD, hidden),
               "v_proj.weight": d.matrix(nkv * HEAD, hidden), "o_proj.weight": d.matrix(hidden, nq * HEAD),
               "q_norm.weight": d.vector(HEAD), "k_norm.weight": d.vector(HEAD)}
    new, past = _numbers(case["new"]), _numbers(case["past"])
    x = d.normal(sum(new), hidden, dtype=torch.bfloat16)
    pages = [-(-(n + p) // PAGE) for n, p in zip(new, past)]
    order = torch.randperm(sum(pages), generator=d.gen, device=DEVICE).to(torch.int32)  # a live cache hands pages out in any order
    table = torch.zeros((len(new), max(pages)), dtype=torch.int32, device=DEVICE)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    shape = (sum(pages), nkv, PAGE, HEAD)
    if any(past):
        k, v = d.normal(*shape, dtype=torch.bfloat16), d.normal(*shape, std=0.02 * hidden ** 0.5, dtype=torch.bfloat16)
    else:
        k, v = (torch.zeros(shape, dtype=torch.bfloat16, device=DEVICE) for _ in range(2))
    return tensors, x, new, past, table, k, v


def _mlp_inputs(case, seed):
    hidden, _, _, ff = LAYERS[case["layer"]]
    d = _Draws(seed)
    tensors = {"gate_proj.weight": d.matrix(ff, hidden), "up_proj.weight": d.matrix(ff, hidden), "down_proj.weight": d.matrix(hidden, ff)}
    return tensors, d.normal(case["tokens"], hidden, dtype=torch.bfloat16)


def _delta_inputs(case, seed):
    hidden, heads, taps, rank, dim = case["hidden"], case["heads"], 4, 64, 128
    d = _Draws(seed)
    t = {"q": d.matrix(heads * dim, hidden), "k": d.matrix(heads * dim, hidden), "v": d.matrix(heads * dim, hidden)}
    for name in ("q.conv", "k.conv", "v.conv"):
        t[name] = d.normal(heads * dim, taps, std=0.4)
    t["b"], t["A_log"], t["norm"] = d.matrix(heads, hidden), d.normal(heads, mean=-1.0, std=0.7), d.vector(dim)
    t["a1"], t["a2"], t["dt_bias"] = d.matrix(rank, hidden), d.matrix(heads * dim, rank), d.normal(heads * dim, mean=-1.0)
    t["g1"], t["g2"], t["o"] = d.matrix(rank, hidden), d.matrix(heads * dim, rank), d.matrix(hidden, heads * dim)
    new = _numbers(case["new"])
    return t, d.normal(sum(new), hidden, dtype=torch.bfloat16), new


def _experts_inputs(case, seed):
    hidden, ff, E = case["hidden"], case["ff"], case["experts"]
    d = _Draws(seed)
    gate, up, down = d.matrix(E, ff, hidden), d.matrix(E, ff, hidden), d.matrix(E, hidden, ff)
    router, correction = d.normal(E, hidden, std=0.02), d.normal(E, std=0.3)
    return gate, up, down, router, correction, d.normal(case["tokens"], hidden, dtype=torch.bfloat16)


def _sample_inputs(case, seed):
    d = _Draws(seed)
    return d.normal(case["rows"], case["vocab"], std=2.5), d.ints(1000, case["rows"]), d.ints(500, case["rows"])


def _step(new, past, dtype=torch.bfloat16):
    return plan_step([SequenceStep(i, p, [0] * n, []) for i, (n, p) in enumerate(zip(new, past))], dtype, DEVICE, 1)


# ------------------------------------------------------------------ what a program has in hand, and one pass
def prepare(case, seed):
    kind = case["kind"]
    if kind == "engine":
        cfg, tensors, ids, prompts = _engine_inputs(case, seed)
        config = config_from_dict(cfg)
        dtype = getattr(torch, case["dtype"])
        model = Model(architecture(config.ARCH_NAMES[0]).build_plan(config), config, dtype, DEVICE)
        model.load({name: t.to(dtype) if t.dtype == torch.bfloat16 else t for name, t in tensors.items()})
        longest = sum(-(-len(row) // PAGE) * PAGE for row in ids)
        return {"kind": kind, "engine": Engine(model, longest, max_seqs=len(ids)), "ids": ids, "prompts": prompts, "steps": case["steps"],
                "every": case["dtype"] == "float32"}
    if kind == "attention":
        hidden, nq, nkv, _ = LAYERS[case["layer"]]
        tensors, x, new, past, table, k, v = _attention_inputs(case, seed)
        rope = build_part("position", "rope", dim=HEAD, base=ROPE_BASE)
        part = build_part("mixer", "gqa_attention", hidden_size=hidden, n_q_heads=nq, n_kv_heads=nkv, head_dim=HEAD, qk_norm_eps=EPS, position=rope)
        part.load(tensors)
        ctx = _step(new, past)
        rope.prepare(ctx.max_position, DEVICE)
        return {"kind": kind, "part": part, "x": x, "ctx": ctx, "cache": PagedKV(k, v, table, DecodeWork(DEVICE))}
    if kind == "mlp":
        hidden, _, _, ff = LAYERS[case["layer"]]
        tensors, x = _mlp_inputs(case, seed)
        part = build_part("feed_forward", "swiglu", hidden_size=hidden, intermediate_size=ff)
        part.load(tensors)
        return {"kind": kind, "part": part, "x": x, "ctx": _step([1] * case["tokens"] if case["tokens"] <= 64 else [case["tokens"]],
                                                                 [0] * case["tokens"] if case["tokens"] <= 64 else [0])}
    if kind == "delta":
        tensors, x, new = _delta_inputs(case, seed)
        part = build_part("mixer", "channel_delta", hidden_size=case["hidden"], n_heads=case["heads"], n_kv_heads=case["heads"], key_dim=128,
                          value_dim=128, conv_taps=4, norm_eps=EPS)
        part.load(tensors)
        cache = tuple(torch.zeros((len(new), *r.shape), dtype=r.dtype, device=DEVICE) for r in part.cache_request())
        return {"kind": kind, "part": part, "x": x, "ctx": _step(new, [0] * len(new)), "cache": cache}
    if kind == "experts":
        gate, up, down, router, correction, x = _experts_inputs(case, seed)
        part = build_part("feed_forward", "routed_experts", hidden_size=case["hidden"], expert_size=case["ff"], n_experts=case["experts"],
                          top=case["top"], n_groups=case["groups"], keep_groups=case["keep"])
        tensors = {"router": router, "correction": correction}
        for e in range(case["experts"]):
            tensors.update({f"e{e}.gate": gate[e], f"e{e}.up": up[e], f"e{e}.down": down[e]})
        part.load(tensors)
        return {"kind": kind, "part": part, "x": x, "ctx": _step([1] * case["tokens"], [0] * case["tokens"])}
    logits, requests, steps = _sample_inputs(case, seed)
    return {"kind": kind, "logits": logits, "requests": requests, "steps": steps,
            "params": SamplingParams(temperature=case["temperature"], top_k=case["top_k"] or None, seed=int(seed))}


def run(state):
    kind = state["kind"]
    if kind == "engine":
        engine, ids, prompts = state["engine"], state["ids"], state["prompts"]
        out = [engine.step([StepEntry(i, row[:n], list(range(n)) if state["every"] else [n - 1]) for i, (row, n) in enumerate(zip(ids, prompts))])]
        for s in range(state["steps"]):
            out.append(engine.step([StepEntry(i, [row[n + s]], [0]) for i, (row, n) in enumerate(zip(ids, prompts))]))
        engine.end_all()
        return out
    if kind == "attention":
        return [state["part"].forward(state["x"], state["ctx"], state["cache"]), state["cache"].k, state["cache"].v]
    if kind == "delta":
        return [state["part"].forward(state["x"], state["ctx"], state["cache"]), *state["cache"]]
    if kind in ("mlp", "experts"):
        return state["part"].forward(state["x"], state["ctx"])
    return choose(state["logits"], state["params"], state["requests"], state["steps"])


# ------------------------------------------------------------------ the work that the path cannot do without
def _attended(new, past):
    return sum(n * p + n * (n + 1) // 2 for n, p in zip(new, past))


def work(case):
    kind = case["kind"]
    if kind == "engine":
        cfg = MODELS[case["model"]]
        size = 4 if case["dtype"] == "float32" else 2
        h, ff, dim, nl = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"], cfg["num_hidden_layers"]
        nq, nkv, vocab = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["vocab_size"]
        layer = h * (2 * nq + 2 * nkv) * dim + 3 * h * ff
        prompts, steps = _numbers(case["prompts"]), case["steps"]
        tokens = sum(prompts) + len(prompts) * steps
        logits = (sum(prompts) if case["dtype"] == "float32" else len(prompts)) + len(prompts) * steps
        kv = 2 * nkv * dim * nl * size
        cached = sum(steps * n + steps * (steps - 1) // 2 for n in prompts) * kv + tokens * kv
        attended = sum((n + steps) * (n + steps + 1) // 2 for n in prompts)
        return {"bytes": (steps + 1) * (nl * layer + vocab * h) * size + cached + logits * vocab * 4,
                "flops": 2 * tokens * nl * layer + 2 * logits * vocab * h + 4 * attended * nq * dim * nl}
    if kind == "attention":
        hidden, nq, nkv, _ = LAYERS[case["layer"]]
        new, past = _numbers(case["new"]), _numbers(case["past"])
        weights, t = hidden * (2 * nq + 2 * nkv) * HEAD, sum(new)
        return {"bytes": 2 * (weights + 2 * t * hidden + 2 * nkv * HEAD * (sum(past) + t)),
                "flops": 2 * t * weights + 4 * _attended(new, past) * nq * HEAD}
    if kind == "mlp":
        hidden, _, _, ff = LAYERS[case["layer"]]
        return {"bytes": 2 * (3 * hidden * ff + 2 * case["tokens"] * hidden), "flops": 6 * case["tokens"] * hidden * ff}
    if kind == "delta":
        hidden, heads, t = case["hidden"], case["heads"], sum(_numbers(case["new"]))
        wide = heads * 128
        weights = 4 * hidden * wide + heads * hidden + 2 * 64 * (hidden + wide)
        states = 2 * len(_numbers(case["new"])) * (heads * 128 * 128 + 3 * 3 * wide) * 4
        return {"bytes": 2 * weights + 4 * t * hidden + states, "flops": 2 * t * weights + 7 * t * heads * 128 * 128}
    if kind == "experts":
        hidden, ff, E, t = case["hidden"], case["ff"], case["experts"], case["tokens"]
        distinct = E * (1 - (1 - case["top"] / E) ** t)  # experts that uniform choices of t tokens touch
        return {"bytes": int(distinct * 6 * hidden * ff) + 4 * E * hidden + t * hidden * 6,
                "flops": 6 * t * case["top"] * hidden * ff + 2 * t * E * hidden}
    n = case["rows"] * case["vocab"]
    return {"bytes": 4 * n + 4 * case["rows"], "flops": 2 * n}


def tolerance(case):
    """About four times what the path differs by from the same formulas with other sums: 32-bit sums, or one rounding to
    bfloat16 here and there in a layer; the whole bfloat16 model carries such roundings through 28 layers."""
    kind = case["kind"]
    if kind == "sample":
        return "exact"
    if kind == "engine":
        return {"rel": 1e-5, "max": 2e-4} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.3}
    return {"rel": 0.01, "max": 0.1}


# ------------------------------------------------------------------ the same in 64 bits
def _norm(x, weight, eps):
    return x / (x.pow(2).mean(-1, keepdim=True) + eps).sqrt() * weight


def _rotate(x, positions, base):
    """x [T, heads, dim]; the angle is defined as a 32-bit product of position and frequency."""
    dim = x.shape[-1]
    inv = 1.0 / (base ** (torch.arange(0, dim, 2, dtype=torch.float32) / dim)).to(x.device)
    angle = (positions.float()[:, None] * inv[None, :]).double()[:, None, :]
    a, b = x[..., :dim // 2], x[..., dim // 2:]
    return torch.cat([a * angle.cos() - b * angle.sin(), b * angle.cos() + a * angle.sin()], dim=-1)


def _attend(q, k, v, past):
    """q [T, nq, d] after ``past`` cached tokens over k, v [past + T, nkv, d], head by head."""
    group, T = q.shape[1] // k.shape[1], q.shape[0]
    out = torch.empty_like(q)
    seen = torch.arange(k.shape[0], device=q.device)[None, :] <= (past + torch.arange(T, device=q.device))[:, None]
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // group].T * q.shape[2] ** -0.5
        out[:, h] = s.masked_fill(~seen, -math.inf).softmax(-1) @ v[:, h // group]
    return out


def _exact_engine(case, seed):
    cfg, t, ids, prompts = _engine_inputs(case, seed)
    nq, nkv, dim, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    rows = []
    for row in ids:
        tokens, pos = torch.tensor(row, device=DEVICE), torch.arange(len(row), device=DEVICE)
        h = t["model.embed_tokens.weight"][tokens].double()
        for i in range(cfg["num_hidden_layers"]):
            w = lambda name: t[f"model.layers.{i}.{name}.weight"].double()
            x = _norm(h, w("input_layernorm"), eps)
            q = _norm((x @ w("self_attn.q_proj").T).view(-1, nq, dim), w("self_attn.q_norm"), eps)
            k = _norm((x @ w("self_attn.k_proj").T).view(-1, nkv, dim), w("self_attn.k_norm"), eps)
            v = (x @ w("self_attn.v_proj").T).view(-1, nkv, dim)
            o = _attend(_rotate(q, pos, cfg["rope_theta"]), _rotate(k, pos, cfg["rope_theta"]), v, 0)
            h = h + o.reshape(len(row), -1) @ w("self_attn.o_proj").T
            x = _norm(h, w("post_attention_layernorm"), eps)
            h = h + (torch.nn.functional.silu(x @ w("mlp.gate_proj").T) * (x @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T
        head = t["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]
        rows.append(_norm(h, t["model.norm.weight"].double(), eps) @ head.double().T)
    every = case["dtype"] == "float32"
    out = [torch.cat([r[:n] if every else r[n - 1:n] for r, n in zip(rows, prompts)])]
    return out + [torch.stack([r[n + s] for r, n in zip(rows, prompts)]) for s in range(case["steps"])]


def _exact_attention(case, seed):
    hidden, nq, nkv, _ = LAYERS[case["layer"]]
    t, x, new, past, table, k_pages, v_pages = _attention_inputs(case, seed)
    x, k_pages, v_pages = x.double(), k_pages.double(), v_pages.double()
    q_all = _norm((x @ t["q_proj.weight"].double().T).view(-1, nq, HEAD), t["q_norm.weight"].double(), EPS)
    k_all = _norm((x @ t["k_proj.weight"].double().T).view(-1, nkv, HEAD), t["k_norm.weight"].double(), EPS)
    v_all = (x @ t["v_proj.weight"].double().T).view(-1, nkv, HEAD)
    o, at = torch.empty_like(q_all), 0
    for i, (n, p) in enumerate(zip(new, past)):
        pos = torch.arange(p, p + n, device=DEVICE)
        page, place = table[i, pos // PAGE].long(), pos % PAGE
        k_pages[page, :, place] = _rotate(k_all[at:at + n], pos, ROPE_BASE)
        v_pages[page, :, place] = v_all[at:at + n]
        seen = torch.arange(p + n, device=DEVICE)
        page, place = table[i, seen // PAGE].long(), seen % PAGE
        o[at:at + n] = _attend(_rotate(q_all[at:at + n], pos, ROPE_BASE), k_pages[page, :, place], v_pages[page, :, place], p)
        at += n
    return [o.reshape(len(x), -1) @ t["o_proj.weight"].double().T, k_pages, v_pages]


def _exact_delta(case, seed):
    t, x, new = _delta_inputs(case, seed)
    t = {name: w.double() for name, w in t.items()}
    x, heads, dim, taps = x.double(), case["heads"], 128, 4
    raw = torch.cat([x @ t[n].T for n in ("q", "k", "v")], dim=1)
    beta = (x @ t["b"].T).sigmoid()
    decay = torch.exp(-t["A_log"].exp()[:, None] * torch.nn.functional.softplus(x @ t["a1"].T @ t["a2"].T + t["dt_bias"]).view(-1, heads, dim))
    conv = torch.cat([t["q.conv"], t["k.conv"], t["v.conv"]])
    outs, states, rings, at = [], [], [], 0
    for n in new:
        mine = torch.cat([raw.new_zeros(taps - 1, raw.shape[1]), raw[at:at + n]])
        y = torch.nn.functional.silu(sum(mine[j:j + n] * conv[:, j] for j in range(taps)))
        q, k, v = (part.reshape(n, heads, dim) for part in y.chunk(3, dim=1))
        q = q / (q.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt() * dim ** -0.5
        k = k / (k.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
        S = x.new_zeros(heads, dim, dim)
        o = torch.empty_like(v)
        for i in range(n):
            S = S * decay[at + i][:, :, None]
            u = beta[at + i][:, None] * (v[i] - (k[i][:, None, :] @ S)[:, 0])
            S = S + k[i][:, :, None] * u[:, None, :]
            o[i] = (q[i][:, None, :] @ S)[:, 0]
        outs.append(o)
        states.append(S)
        rings.append(mine[n:])
        at += n
    o = _norm(torch.cat(outs), t["norm"], EPS) * (x @ t["g1"].T @ t["g2"].T).sigmoid().view(-1, heads, dim)
    return [o.reshape(len(x), -1) @ t["o"].T, torch.stack(states), torch.stack(rings)]


def _exact_experts(case, seed):
    gate, up, down, router, correction, x = _experts_inputs(case, seed)
    x, E, groups = x.double(), case["experts"], case["groups"]
    s = (x @ router.double().T).sigmoid()
    choice = s + correction.double()
    score = choice.view(-1, groups, E // groups).topk(2, dim=-1).values.sum(-1)
    kept = torch.zeros_like(score, dtype=torch.bool).scatter_(1, score.topk(case["keep"], dim=1).indices, True)
    chosen = choice.masked_fill(~kept.repeat_interleave(E // groups, dim=1), -math.inf).topk(case["top"], dim=1).indices
    out = torch.zeros_like(x)
    for e in range(E):
        rows, _ = (chosen == e).nonzero(as_tuple=True)
        if len(rows):
            y = x[rows]
            act = torch.nn.functional.silu(y @ gate[e].double().T) * (y @ up[e].double().T)
            out[rows] += s[rows, e][:, None] * (act @ down[e].double().T)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "engine":
        return _exact_engine(case, seed)
    if kind == "attention":
        return _exact_attention(case, seed)
    if kind == "mlp":
        t, x = _mlp_inputs(case, seed)
        t, x = {name: w.double() for name, w in t.items()}, x.double()
        return (torch.nn.functional.silu(x @ t["gate_proj.weight"].T) * (x @ t["up_proj.weight"].T)) @ t["down_proj.weight"].T
    if kind == "delta":
        return _exact_delta(case, seed)
    if kind == "experts":
        return _exact_experts(case, seed)
    return None
