"""Routed experts whose weights come in boxes through rings: rows shorter than a box, odd numbers of pieces a warp, rows that leave room for one block
an SM and for the small rings, runs of one and of many tokens an expert."""

import pytest
import torch

from tests.test_gpu_kernels import DEV, F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,width,ff,experts,top", [
    (700, 64, 32, 8, 6), (512, 96, 160, 8, 4), (300, 224, 96, 5, 5), (40, 2048, 64, 16, 4), (24, 4096, 128, 3, 2), (9, 6144, 160, 4, 3), (8, 9216, 64, 4, 4),
    (16, 96, 9216, 3, 2), (63, 512, 2048, 16, 4), (63, 1024, 768, 32, 4), (30, 2048, 1024, 8, 3)])
def test_rows_of_every_length(tokens, width, ff, experts, top):
    gen = torch.Generator(device=DEV).manual_seed(width + ff)
    draw = lambda *shape, scale=1.0: torch.randn(shape, generator=gen, device=DEV) * scale
    h = draw(tokens, width).bfloat16()
    gate_up, down = draw(experts, 2, ff, width, scale=width**-0.5).bfloat16(), draw(experts, width, ff, scale=ff**-0.5).bfloat16()
    ids = draw(tokens, experts).topk(top, dim=1).indices.int().contiguous()
    weights = draw(tokens, top).abs()
    got = F().experts_pairwise(h, gate_up, down, ids, weights, None, None).double()
    F().check_kernel_errors(DEV)
    want, bound = torch.zeros_like(got), torch.zeros_like(got)
    for e in range(experts):
        rows, place = (ids == e).nonzero(as_tuple=True)
        if not len(rows):
            continue
        z, u = (h[rows].double() @ gate_up[e, i].double().T for i in (0, 1))
        act = torch.nn.functional.silu(z) * u
        w = weights[rows, place].double()[:, None]
        want.index_add_(0, rows, w * (act @ down[e].double().T))
        # inner values are rounded to bfloat16; 32-bit sums of `width` and `ff` terms
        spread = act.abs() * 2.0**-8 + 2.0**-23 * width**0.5 * (h[rows].double().abs() @ gate_up[e, 0].double().abs().T) * (1 + u.abs())
        bound.index_add_(0, rows, w * (spread @ down[e].double().abs().T + 2.0**-23 * ff**0.5 * (act.abs() @ down[e].double().abs().T)))
    assert ((got - want).abs() <= bound + 1e-6).all()
