"""Launches that overlap the end of their predecessor may not change a bit of what a step computes."""
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD, Config, PowerSGD, optimizer_step

pytestmark = pytest.mark.gpu

SHAPES = [(64, 3, 3, 3), (64, 576), (64, 576), (130, 650), (300, 1201), (512, 2304), (10, 512), (2049, 260)]


def _gradients(shapes, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(s, generator=g, device="cuda") for s in shapes]


def _aggregate(shapes, rank, iters, prepare=None):
    core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=rank, num_iters_per_step=iters), backend="native")
    grads, seen = _gradients(shapes, 0), []
    for step in range(4):
        if step and prepare is not None:
            prepare(core._native)
        seen += [o.clone() for o in core.aggregate(grads)] + [g.clone() for g in grads]
        torch._foreach_add_(grads, _gradients(shapes, 1 + step))   # no pause: the next step starts behind this
    return seen + [core._ps_buffer, core._qs_buffer], core._native


@pytest.mark.parametrize("rank,iters", [(1, 2), (2, 2), (4, 1), (4, 3), (16, 2)])
def test_overlapped_launches_leave_the_bits_alone(rank, iters):
    usual, native = _aggregate(SHAPES, rank, iters)
    assert native._chained()
    apart, _ = _aggregate(SHAPES, rank, iters, lambda nat: setattr(nat, "_chained", lambda: False))
    for a, b in zip(usual, apart):
        assert torch.equal(a, b)


def test_tensor_core_products_behind_an_overlapped_basis():
    shapes = [(1024, 1100), (2176, 900)]
    usual, native = _aggregate(shapes, 8, 2)
    assert native.uses_tensor_cores
    apart, _ = _aggregate(shapes, 8, 2, lambda nat: setattr(nat, "_chained", lambda: False))
    assert all(torch.equal(a, b) for a, b in zip(usual, apart))


def test_recorded_in_a_graph_and_run_eagerly_agree():
    shapes = [(128, 300), (70, 129), (33,)]

    def run(record):
        params = [torch.nn.Parameter(x) for x in _gradients(shapes, 9)]
        for p, x in zip(params, _gradients(shapes, 10)):
            p.grad = x
        opt = torch.optim.SGD(params, lr=0.1, momentum=0.9)
        agg = PowerSGD(params, Config(rank=2, num_iters_per_step=2, start_compressing_after_num_steps=0))
        fresh = _gradients(shapes, 11)

        def step():
            torch._foreach_add_([p.grad for p in params], fresh)
            optimizer_step(opt, agg)

        step()
        if record:
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                step()
            for _ in range(4):
                graph.replay()
        else:
            for _ in range(4):
                step()
        torch.cuda.synchronize()
        return [t.clone() for p in params for t in (p.detach(), p.grad)]

    for a, b in zip(run(True), run(False)):
        assert torch.equal(a, b)
