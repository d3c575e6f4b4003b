"""Which kernels may start before the one in front has finished: by the switch, by the thread, by the engine's option."""

import ctypes
import threading

import pytest
import torch

from gtar_kimik3_public_b200.ops.functional import set_pdl
from gtar_kimik3_public_b200.ops.library import in_order, library, one_layer


def test_the_switch_has_three_settings():
    before = set_pdl(None)
    try:
        assert set_pdl(True) is None and set_pdl(False) is True and set_pdl(None) is False and set_pdl(None) is None
    finally:
        set_pdl(before)


def test_a_thread_in_order_stays_so_within_layers_and_alone():
    chain, seen, other = library().gk_chain, [], []

    @one_layer
    def layer():
        seen.append(chain(-1))

    @in_order
    def step():
        layer()
        seen.append(chain(-1))
        thread = threading.Thread(target=lambda: other.append(chain(0)))
        thread.start()
        thread.join()

    step()
    assert seen == [-1, -1] and other == [0] and chain(0) == 0


def _early_edges(run):
    """How many of a capture's kernels stand behind another one, and how many of these may start before it has finished."""
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        run()
    get = ctypes.CDLL("libcuda.so.1").cuGraphGetEdges_v2
    handle, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert get(handle, None, None, None, ctypes.byref(count)) == 0
    n = count.value
    ends, data = [(ctypes.c_void_p * n)() for _ in range(2)], (ctypes.c_ubyte * (8 * n))()  # of an edge: from_port, to_port, type, ..
    assert get(handle, *ends, data, ctypes.byref(count)) == 0
    return n, sum(data[8 * i + 2] == 1 for i in range(n))


@pytest.mark.gpu
def test_captured_layers_by_the_switch_and_the_thread():
    from gtar_kimik3_public_b200.engine.step import SequenceStep, plan_step
    from gtar_kimik3_public_b200.parts.base import build_part
    from tests.test_gpu_kernels import DEV, rand

    b = lambda *shape: rand(*shape, seed=sum(shape), scale=0.05).to(torch.bfloat16).to(DEV)
    part = build_part("feed_forward", "routed_experts", hidden_size=1024, expert_size=768, n_experts=4, top=2)
    tensors = {"router": b(4, 1024).float(), "correction": b(4).float()}
    for e in range(4):
        tensors.update({f"e{e}.gate": b(768, 1024), f"e{e}.up": b(768, 1024), f"e{e}.down": b(1024, 768)})
    part.load(tensors)
    x = b(32, 1024)
    ctx = plan_step([SequenceStep(i, 0, [0], []) for i in range(32)], torch.bfloat16, torch.device(DEV), 1)
    run = lambda: part.forward(x, ctx)
    run()
    torch.cuda.synchronize()
    default, thread = _early_edges(run), _early_edges(in_order(run))
    before = set_pdl(False)
    try:
        off = _early_edges(run)
    finally:
        set_pdl(before)
    assert default[0] > 2 and default == (default[0], default[0])  # all behind the first
    assert thread == off == (default[0], 0)


@pytest.mark.gpu
@pytest.mark.parametrize("graphs", [True, False])
def test_an_engine_without_early_launches_has_none(monkeypatch, tmp_path, graphs):
    """The thread's state as the model's steps see it, captured and not; and the switch is afterwards what it was."""
    from gtar_kimik3_public_b200 import generate as api
    from gtar_kimik3_public_b200.engine.engine import Engine, StepEntry
    from gtar_kimik3_public_b200.registry import config_from_dict
    from gtar_kimik3_public_b200.weights import write_random_model
    from tests.tiny_configs import TINY_B

    write_random_model(tmp_path, config_from_dict(TINY_B), seed=0, std=0.08)
    model = api.load(tmp_path, "bfloat16", "cuda:0")
    chain, seen, step = library().gk_chain, [], model.step

    def watched(*args):
        state = chain(0)
        chain(state)
        seen.append(state)
        return step(*args)

    monkeypatch.setattr(model, "step", watched)
    before = set_pdl(None)
    set_pdl(before)
    results = []
    for use_pdl in (False, True):
        engine = Engine(model, 256, use_graphs=graphs, use_pdl=use_pdl)
        seen.clear()
        results.append([engine.step([StepEntry(0, [1, 2, 3], [2])]).clone(), *(engine.step([StepEntry(0, [4], [0])]).clone() for _ in range(3))])
        assert seen and set(seen) == {0 if use_pdl else -1}
    assert all(torch.equal(a, b) for a, b in zip(*results))
    after = set_pdl(before)
    assert after is before and chain(0) == 0
