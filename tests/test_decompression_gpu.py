"""The decompression with error feedback and update against float64 at the edges of its strips."""
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD, Config, PowerSGD, optimizer_step
from powersgd_b200.cuda_path import NativeCompressor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank,iters", [(2, 1), (4, 2), (8, 2), (16, 1), (11, 2), (16, 2)])
@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_decompression_and_update_at_strip_edges(rank, iters, momentum):
    """Residual and update of one step in float64 from the factors the launches used (at most 32 products
    per entry, each side rounded to float32): off by at most about (K + 3) 2^-24 of the terms' sizes."""
    shapes = [s for s in [(40, 66), (95, 130), (97, 129), (161, 512), (300, 260), (64, 257)]]
    g = torch.Generator(device="cuda").manual_seed(5)
    draw = lambda s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    params = [torch.nn.Parameter(draw(s)) for s in shapes]
    opt = torch.optim.SGD(params, lr=0.1, momentum=momentum)
    for p in params:
        p.grad = draw(p.shape)
        if momentum:
            opt.state[p]["momentum_buffer"] = draw(p.shape)
    before = [(p.detach().double().clone(), p.grad.double().clone(), opt.state[p]["momentum_buffer"].double().clone() if momentum else None) for p in params]
    agg = PowerSGD(params, Config(rank=rank, min_compression_rate=0.1, num_iters_per_step=iters, start_compressing_after_num_steps=0))
    optimizer_step(opt, agg)
    core, nat = agg._powersgd, agg._powersgd._native
    for grp in core.plan.groups:
        for pos, idx in enumerate(grp.members):
            p0, q0 = grp.p_offset + pos * grp.n * grp.r, grp.q_offset + pos * grp.m * grp.r
            cut = lambda buf, at, rows: buf[at : at + rows * grp.r].view(rows, grp.r).double()  # noqa: E731
            update = size = 0.0
            for t in range(iters):
                left, right = (nat.h_in[t], nat.h_loc[t]) if t % 2 == 0 else (nat.h_loc[t], nat.h_in[t])
                L, R = cut(left, p0, grp.n), cut(right, q0, grp.m)
                update, size = update + L @ R.T, size + L.abs() @ R.abs().T
            p, grad, mom = before[idx]
            p, grad = p.view(grp.n, grp.m), grad.view(grp.n, grp.m)
            eps = (grp.r * iters + 3) * 2.0 ** -24
            now = params[idx]
            assert ((now.grad.double().view_as(grad) - (grad - update)).abs() <= eps * (size + grad.abs())).all(), shapes[idx]
            v = update if mom is None else momentum * mom.view_as(p) + update
            bound = eps * (size + (0 if mom is None else mom.view_as(p).abs()))
            if mom is not None:
                assert ((opt.state[now]["momentum_buffer"].double().view_as(p) - v).abs() <= bound).all(), shapes[idx]
            assert ((now.detach().double().view_as(p) - (p - 0.1 * v)).abs() <= bound + 2.0 ** -23 * (p.abs() + v.abs())).all(), shapes[idx]


@pytest.mark.parametrize("rank,rows", [(8, 256), (16, 256), (16, 96)])
def test_local_and_summed_factors_apart(rank, rows):
    """What several workers run (there without a channel): the residual from the local factors, the update
    from the summed ones, in strips up to the tallest. The same bound as above, per product."""
    shapes, iters, workers = [(700, 300), (256, 129), (97, 66)], 2, 3
    core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=rank, num_iters_per_step=iters), backend="native")
    g = torch.Generator(device="cuda").manual_seed(rank)
    draw = lambda s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    grads = [draw(s) for s in shapes]
    core.aggregate(grads)
    nat = core._native
    assert int(nat.lib.psgd_finalize_strip_rows(iters * rank, 0)) == 256
    nat.tiles.fin_rows, nat._key = rows, None
    nat._bind(grads)
    for buf in nat.h_in + nat.h_loc + nat.h_sum:
        buf.copy_(draw(buf.shape))
    before = [x.double().clone() for x in grads]
    nat._finalize([True, False], False, workers)
    for grp in core.plan.groups:
        for pos, idx in enumerate(grp.members):
            p0, q0 = grp.p_offset + pos * grp.n * grp.r, grp.q_offset + pos * grp.m * grp.r
            cut = lambda buf, at, n: buf[at : at + n * grp.r].view(n, grp.r).double()  # noqa: E731
            own = [(cut(nat.h_in[0], p0, grp.n), cut(nat.h_loc[0], q0, grp.m)), (cut(nat.h_loc[1], p0, grp.n), cut(nat.h_in[1], q0, grp.m))]
            all_ = [(cut(nat.h_in[0], p0, grp.n), cut(nat.h_sum[0], q0, grp.m)), (cut(nat.h_sum[1], p0, grp.n), cut(nat.h_in[1], q0, grp.m))]
            product = lambda pairs: (sum(l @ r.T for l, r in pairs), sum(l.abs() @ r.abs().T for l, r in pairs))  # noqa: E731
            eps, was = (grp.r * iters + 3) * 2.0 ** -24, before[idx]
            (mine, mine_size), (total, total_size) = product(own), product(all_)
            assert ((grads[idx].double() - (was - mine)).abs() <= eps * (mine_size + was.abs())).all(), shapes[idx]
            assert ((nat._out_views[idx].double() - total / workers).abs() <= eps * total_size / workers).all(), shapes[idx]


@pytest.mark.parametrize("rank,iters", [(8, 2), (8, 3), (12, 2), (16, 1), (16, 2)])
@pytest.mark.parametrize("first", [(64, 48), (5, 9)])
def test_left_panels_by_rows(rank, iters, first, monkeypatch):
    """From 16 factor columns on: factors on 16-byte boundaries and, behind a matrix of rank 5, not. The bound of the first test."""
    monkeypatch.setattr(NativeCompressor, "STRIPS_BY_16", 0.0)
    shapes = [first, (97, 129), (300, 260), (257, 66), (520, 128)]
    core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=rank, num_iters_per_step=iters), backend="native")
    g = torch.Generator(device="cuda").manual_seed(rank)
    grads = [torch.randn(s, generator=g, device="cuda") for s in shapes]
    before = [x.double() for x in grads]
    outs, nat = core.aggregate(grads), core._native
    for grp in core.plan.groups:
        for pos, idx in enumerate(grp.members):
            p0, q0 = grp.p_offset + pos * grp.n * grp.r, grp.q_offset + pos * grp.m * grp.r
            cut = lambda buf, at, n: buf[at : at + n * grp.r].view(n, grp.r).double()  # noqa: E731
            pairs = [(cut(a, p0, grp.n), cut(b, q0, grp.m)) for a, b in
                     ((nat.h_in[t], nat.h_loc[t]) if t % 2 == 0 else (nat.h_loc[t], nat.h_in[t]) for t in range(iters))]
            update, size = sum(l @ r.T for l, r in pairs), sum(l.abs() @ r.abs().T for l, r in pairs)
            eps = (grp.r * iters + 3) * 2.0 ** -24
            assert ((outs[idx].double() - update).abs() <= eps * size).all(), shapes[idx]
            assert ((grads[idx].double() - (before[idx] - update)).abs() <= eps * (size + before[idx].abs())).all(), shapes[idx]


@pytest.mark.parametrize("shapes,flags", [([(300, 260), (64, 48)], 4), ([(300, 260), (64, 49)], 0), ([(300, 261)], 0), ([(900, 1024), (64, 49)], 4)])
def test_strips_by_rows_are_for_lists_that_gain(shapes, flags):
    core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=8, num_iters_per_step=2), backend="native")
    core.aggregate([torch.randn(s, device="cuda") for s in shapes])
    assert core._native._strip_flags == flags
