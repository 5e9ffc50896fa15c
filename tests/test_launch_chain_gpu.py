"""Launches that overlap the end of their predecessor, and steps repeated from their recorded calls:
neither may change a bit of what a step computes."""
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
def test_overlapped_and_repeated_launches_leave_the_bits_alone(rank, iters):
    usual, native = _aggregate(SHAPES, rank, iters)
    assert native._chained() and native._tapes
    apart, _ = _aggregate(SHAPES, rank, iters, lambda nat: (setattr(nat, "_chained", lambda: False), nat._tapes.clear()))
    again, _ = _aggregate(SHAPES, rank, iters, lambda nat: nat._tapes.clear())
    for a, b, c in zip(usual, apart, again):
        assert torch.equal(a, b) and torch.equal(a, c)


def test_tensor_core_products_behind_an_overlapped_basis():
    shapes = [(1024, 1100), (2176, 900)]
    usual, native = _aggregate(shapes, 8, 2)
    assert native.uses_tensor_cores
    apart, _ = _aggregate(shapes, 8, 2, lambda nat: (setattr(nat, "_chained", lambda: False), nat._tapes.clear()))
    assert all(torch.equal(a, b) for a, b in zip(usual, apart))


def test_new_gradients_new_rates_and_new_factors_are_seen():
    """What a repeated step must not take from the step it repeats: the tensors, the learning rate, the
    factors that a checkpoint put in place."""
    def make():
        g = torch.Generator(device="cuda").manual_seed(3)
        params = [torch.nn.Parameter(torch.randn(s, generator=g, device="cuda")) for s in [(96, 200), (96, 200), (50, 40), (33,)]]
        opt = torch.optim.SGD(params, lr=0.1, momentum=0.9)
        return params, opt, PowerSGD(params, Config(rank=2, num_iters_per_step=2, start_compressing_after_num_steps=0))

    (pa, oa, aa), (pb, ob, ab) = make(), make()
    for step in range(8):
        fresh = _gradients([tuple(p.shape) for p in pa], 40 + step)
        for params, opt, agg in ((pa, oa, aa), (pb, ob, ab)):
            if step in (0, 5):   # tensors of their own from here on
                for p, f in zip(params, fresh):
                    p.grad = f.clone() if p.grad is None else p.grad + f
            else:
                torch._foreach_add_([p.grad for p in params], fresh)
            opt.param_groups[0]["lr"] = 0.1 / (1 + step // 3)
            if step == 6:
                for view in agg._powersgd._ps + agg._powersgd._qs:
                    view.copy_(torch.ones_like(view).cumsum(1).sin())
            if agg is ab and getattr(agg._powersgd, "_native", None) is not None:
                agg._powersgd._native._tapes.clear()
                agg._fused._last_values = None
            optimizer_step(opt, agg)
        for p, q in zip(pa, pb):
            assert torch.equal(p, q) and torch.equal(p.grad, q.grad), step


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


def test_loaded_optimizer_state_is_used():
    """`optimizer.load_state_dict` puts other momentum buffers in place; the steps after it update those."""
    import copy

    def run(new_driver):
        params = [torch.nn.Parameter(x) for x in _gradients([(128, 300), (70, 129), (33,)], 9)]
        opt = torch.optim.SGD([{"params": params[:1]}, {"params": params[1:], "lr": 0.05}], lr=0.1, momentum=0.9)
        agg = PowerSGD(params, Config(rank=2, num_iters_per_step=2, start_compressing_after_num_steps=0))
        saved = None
        for i in range(6):
            for p, x in zip(params, _gradients([tuple(p.shape) for p in params], 20 + i)):
                p.grad = x if p.grad is None else p.grad.add_(x)
            if i == 2:
                saved = copy.deepcopy(opt.state_dict())
            if i == 4:
                opt.load_state_dict(saved)
            if new_driver:
                agg._fused = None
            optimizer_step(opt, agg)
        return [t.detach().clone() for p in params for t in (p, p.grad, opt.state[p]["momentum_buffer"])]

    for a, b in zip(run(False), run(True)):
        assert torch.equal(a, b)
