"""Layers called one by one, where the kernels behind a layer's first may start early: many times back to back, with inputs and states that a
kernel in front rewrites in place, they give what they give with every kernel waiting for the one in front."""

import pytest
import torch

from gtar_kimik3_public_b200.engine.step import SequenceStep, plan_step
from gtar_kimik3_public_b200.ops.library import in_order
from gtar_kimik3_public_b200.parts.base import build_part
from tests.test_gpu_kernels import DEV, F, rand

pytestmark = pytest.mark.gpu
TURNS = 12


def b(*shape, scale=0.05):
    return rand(*shape, seed=sum(shape), scale=scale).to(torch.bfloat16).to(DEV)


def mlp(hidden, ff):
    part = build_part("feed_forward", "swiglu", hidden_size=hidden, intermediate_size=ff)
    part.load({"gate_proj.weight": b(ff, hidden), "up_proj.weight": b(ff, hidden), "down_proj.weight": b(hidden, ff)})
    return part, hidden, []


def experts(shared):
    part = build_part("feed_forward", "routed_experts", hidden_size=512, expert_size=256, n_experts=8, top=2, **({"shared_size": 256} if shared else {}))
    tensors = {"router": b(8, 512).float(), "correction": b(8).float()}
    for e in range(8):
        tensors.update({f"e{e}.gate": b(256, 512) * (1 + e), f"e{e}.up": b(256, 512), f"e{e}.down": b(512, 256)})
    if shared:
        tensors.update({"shared.gate": b(256, 512), "shared.up": b(256, 512), "shared.down": b(512, 256)})
    part.load(tensors)
    return part, 512, []


def delta(counts):
    part = build_part("mixer", "channel_delta", hidden_size=256, n_heads=2, n_kv_heads=2, key_dim=128, value_dim=128, conv_taps=4, norm_eps=1e-5)
    part.load({"q": b(256, 256), "k": b(256, 256), "v": b(256, 256), "q.conv": b(256, 4), "k.conv": b(256, 4), "v.conv": b(256, 4), "b": b(2, 256),
               "A_log": b(2), "norm": b(128, scale=1.0), "a1": b(64, 256), "a2": b(256, 64), "dt_bias": b(256), "g1": b(64, 256), "g2": b(256, 64),
               "o": b(256, 256)})
    return part, 256, [torch.zeros((len(counts), *r.shape), dtype=r.dtype, device=DEV) for r in part.cache_request()]


def attention(counts):
    part = build_part("mixer", "gqa_attention", hidden_size=512, n_q_heads=4, n_kv_heads=2, head_dim=128, qk_norm_eps=1e-6, position=None)
    part.load({"q_proj.weight": b(512, 512), "k_proj.weight": b(256, 512), "v_proj.weight": b(256, 512), "o_proj.weight": b(512, 512),
               "q_norm.weight": b(128, scale=1.0), "k_norm.weight": b(128, scale=1.0)})
    pages = sum(-(-n // 64) for n in counts)
    k, v = (torch.zeros(pages, 2, 64, 128, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    table, at = torch.zeros(len(counts), max(-(-n // 64) for n in counts), dtype=torch.int32), 0
    for i, n in enumerate(counts):
        table[i, :-(-n // 64)] = torch.arange(at, at + -(-n // 64))
        at += -(-n // 64)
    return part, 512, [F().PagedKV(k, v, table.to(DEV), F().DecodeWork(torch.device(DEV)))]


@pytest.mark.parametrize("make,counts", [
    (lambda c: mlp(1024, 3072), [1] * 8), (lambda c: mlp(1024, 3072), [1] * 40), (lambda c: mlp(512, 1024), [300]),
    (lambda c: experts(False), [1] * 3), (lambda c: experts(False), [1] * 60), (lambda c: experts(True), [1] * 20), (lambda c: experts(True), [400]),
    (delta, [1] * 6), (delta, [30, 5]), (delta, [300, 2]), (attention, [1] * 5), (attention, [90, 20])])
def test_a_layer_is_what_it_is_with_every_kernel_in_order(make, counts):
    part, hidden, state = make(counts)
    ctx = plan_step([SequenceStep(i, 0, [0] * n, []) for i, n in enumerate(counts)], torch.bfloat16, torch.device(DEV), 1)
    inputs = [rand(sum(counts), hidden, seed=50 + t).to(torch.bfloat16).to(DEV) for t in range(TURNS)]
    is_mixer = bool(state)
    cache = tuple(state) if is_mixer and isinstance(state[0], torch.Tensor) else state[0] if is_mixer else None
    kept = [t for t in (state if is_mixer and isinstance(state[0], torch.Tensor) else [cache.k, cache.v] if is_mixer else [])]

    def run(forward):
        for t in kept:
            t.zero_()
        x, outputs = torch.empty_like(inputs[0]), []
        for fresh in inputs:  # a recurrent layer's state goes on from call to call
            x.copy_(fresh)
            outputs.append(forward(x, ctx, cache) if is_mixer else forward(x, ctx))
        outputs.extend(t.clone() for t in kept)
        return outputs

    run(part.forward)
    for got, want in zip(run(part.forward), run(in_order(part.forward))):
        assert torch.equal(got, want)
