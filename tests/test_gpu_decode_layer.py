"""An attention layer over a decode step as one call: what its three kernels give one by one, on the same pages."""

import pytest
import torch

from gtar_kimik3_public_b200.engine.step import SequenceStep, plan_step
from gtar_kimik3_public_b200.ops import attention as attention_ops
from gtar_kimik3_public_b200.ops.linear import linear
from gtar_kimik3_public_b200.parts.base import build_part
from tests.test_gpu_kernels import DEV, F, rand

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,hidden,n_q,n_kv,dim,norm,rope", [
    ([1], 64, 2, 1, 64, True, True), ([70, 1, 300], 1024, 16, 8, 128, True, True), ([65] * 8, 2560, 32, 8, 128, True, True),
    ([200, 3] * 8, 512, 8, 2, 64, False, True), ([40, 900], 256, 4, 4, 128, True, False)])
def test_the_layer_is_its_kernels(lens, hidden, n_q, n_kv, dim, norm, rope):
    position = build_part("position", "rope", dim=dim, base=1e4) if rope else None
    part = build_part("mixer", "gqa_attention", hidden_size=hidden, n_q_heads=n_q, n_kv_heads=n_kv, head_dim=dim, qk_norm_eps=1e-6 if norm else None,
                      position=position)
    b = lambda *shape, seed: rand(*shape, seed=seed, scale=0.05).to(torch.bfloat16).to(DEV)
    tensors = {"q_proj.weight": b(n_q * dim, hidden, seed=1), "k_proj.weight": b(n_kv * dim, hidden, seed=2), "v_proj.weight": b(n_kv * dim, hidden, seed=3),
               "o_proj.weight": b(hidden, n_q * dim, seed=4)}
    if norm:
        tensors.update({"q_norm.weight": 1 + 0.1 * rand(dim, seed=5).float().to(DEV), "k_norm.weight": 1 + 0.1 * rand(dim, seed=6).float().to(DEV)})
    part.load(tensors)
    n, pages = len(lens), -(-max(lens) // 64)
    x = rand(n, hidden, seed=7).to(torch.bfloat16).to(DEV)
    k, v = (rand(n * pages, n_kv, 64, dim, seed=s).to(torch.bfloat16).to(DEV) for s in (8, 9))
    table = torch.randperm(n * pages, generator=torch.Generator().manual_seed(1)).to(torch.int32).view(n, pages).to(DEV)
    ctx = plan_step([SequenceStep(i, m - 1, [0], []) for i, m in enumerate(lens)], torch.bfloat16, torch.device(DEV), 1)
    if rope:
        position.prepare(ctx.max_position, torch.device(DEV))
    caches = [F().PagedKV(k.clone(), v.clone(), table, F().DecodeWork(torch.device(DEV))) for _ in range(2)]
    splits = part._decode_layer_splits(x, ctx, caches[0])
    assert splits == attention_ops.decode_split_count(ctx, n_kv, caches[0])
    got = part.forward(x, ctx, caches[0])
    o = F().attention_decode_fused(linear(x, part.w_qkv), n_q, n_kv, dim, part.q_norm, part.k_norm, part.qk_norm_eps or 1.0, position and position.cos,
                                   position and position.sin, caches[1], ctx.kv_len, ctx.slots, ctx.max_position, part.scale, 0, splits, True)
    assert torch.equal(got, linear(o.view(n, n_q * dim), part.w_o))
    assert torch.equal(caches[0].k, caches[1].k) and torch.equal(caches[0].v, caches[1].v)


def test_other_steps_go_as_before():
    """Runs of several tokens, 32-bit runs and heads that no fast kernel takes have no such call."""
    part = build_part("mixer", "gqa_attention", hidden_size=64, n_q_heads=2, n_kv_heads=1, head_dim=64, qk_norm_eps=None, position=None)
    b = lambda *shape: torch.zeros(shape, dtype=torch.bfloat16, device=DEV)
    part.load({"q_proj.weight": b(128, 64), "k_proj.weight": b(64, 64), "v_proj.weight": b(64, 64), "o_proj.weight": b(64, 128)})
    cache = F().PagedKV(b(2, 1, 64, 64), b(2, 1, 64, 64), torch.zeros(2, 1, dtype=torch.int32, device=DEV), F().DecodeWork(torch.device(DEV)))
    step = lambda counts: plan_step([SequenceStep(i, 0, [0] * c, []) for i, c in enumerate(counts)], torch.bfloat16, torch.device(DEV), 1)
    assert part._decode_layer_splits(b(2, 64), step([1, 1]), cache) == 1
    assert part._decode_layer_splits(b(3, 64), step([2, 1]), cache) == 0
    assert part._decode_layer_splits(b(2, 64).float(), step([1, 1]), cache) == 0
    assert part._decode_layer_splits(b(130)[1:129].view(2, 64), step([1, 1]), cache) == 0  # a row off 16 bytes
