"""The last product and the decompression in one pass over the gradient, against float64 at the edges of its
panels, groups and columns."""
import pytest
import torch

from powersgd_b200 import Config, PowerSGD
from powersgd_b200.cuda_path import NativeCompressor

pytestmark = pytest.mark.gpu

SHAPES = [(5, 23), (70, 27), (64, 576), (129, 650), (33, 1001), (300, 1024), (41, 514), (600, 64), (2500, 24)]


def _check(shapes, rank, iters, monkeypatch):
    """The fresh P, the update and the residual from the factors of the launches before. P sums m products in chains of
    at most 12 and a tree of at most 10 additions, less the corrections of r products each; an update sums K
    products: off by at most that many 2^-24 of the terms' sizes (each side rounds to float32)."""
    monkeypatch.setattr(NativeCompressor, "PANEL_ELEMS", 0)
    gen = torch.Generator(device="cuda").manual_seed(7)
    draw = lambda s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    params = [torch.nn.Parameter(draw(s)) for s in shapes]
    agg = PowerSGD(params, Config(rank=rank, min_compression_rate=0.01, num_iters_per_step=iters, start_compressing_after_num_steps=0))
    for step in range(2 if iters % 2 else 1):   # a step of an odd number that starts on the Q side ends there
        grads = [draw(p.shape) for p in params]
        before = [g.double() for g in grads]
        outs = agg.aggregate(grads)
    core, nat = agg._powersgd, agg._powersgd._native
    torch.cuda.synchronize()
    nat.check()   # no wait inside a kernel ran out
    assert nat._finished and all(agg.is_compressed_mask)
    eps = 2.0 ** -24
    for grp in core.plan.groups:
        for pos, idx in enumerate(grp.members):
            p0, q0, r = grp.p_offset + pos * grp.n * grp.r, grp.q_offset + pos * grp.m * grp.r, grp.r
            cut = lambda buf, at, rows: buf[at : at + rows * r].view(rows, r).double()  # noqa: E731
            grad = before[idx].view(grp.n, grp.m)
            lefts = [cut(nat.h_loc[t] if (iters - 1 - t) % 2 == 0 else nat.h_in[t], p0, grp.n) for t in range(iters)]
            rights = [cut(nat.h_in[t] if (iters - 1 - t) % 2 == 0 else nat.h_loc[t], q0, grp.m) for t in range(iters)]
            basis, fresh = rights[-1], lefts[-1]
            none = torch.zeros_like(fresh)
            taken = sum((l @ (rt.T @ basis) for l, rt in zip(lefts[:-1], rights[:-1])), none)
            size = grad.abs() @ basis.abs() + sum((l.abs() @ (rt.T.abs() @ basis.abs()) for l, rt in zip(lefts[:-1], rights[:-1])), none)
            assert ((fresh - (grad @ basis - taken)).abs() <= (24 + r + iters) * eps * size).all(), ("P", shapes[idx])
            assert torch.equal(core._ps_buffer[p0 : p0 + grp.n * r], nat.h_loc[iters - 1][p0 : p0 + grp.n * r])
            update = sum(l @ rt.T for l, rt in zip(lefts, rights))
            size = sum(l.abs() @ rt.abs().T for l, rt in zip(lefts, rights))
            bound = (r * iters + 3) * eps
            assert ((grads[idx].double().view_as(grad) - (grad - update)).abs() <= bound * (size + grad.abs())).all(), ("residual", shapes[idx])
            assert ((outs[idx].double().view_as(grad) - update).abs() <= bound * size).all(), ("update", shapes[idx])


@pytest.mark.parametrize("rank,iters", [(1, 1), (1, 2), (1, 3), (1, 4), (2, 1), (2, 2), (2, 3), (2, 4), (3, 2), (4, 1), (4, 2), (5, 1), (8, 1)])
def test_one_pass_against_float64(rank, iters, monkeypatch):
    _check(SHAPES + [(37, 4608 if rank * iters <= 4 else 4096)], rank, iters, monkeypatch)


@pytest.mark.parametrize("rank,iters", [(2, 2), (4, 2), (8, 1)])
def test_segments_of_unlike_matrices(rank, iters, monkeypatch):
    """Two or three segments per block, in turn of one group and four rows per panel and of eight groups and up to
    sixteen rows: the rings begin elsewhere in each of them."""
    wide = 4608 if rank * iters <= 4 else 4096
    _check([s for i in range(100) for s in [(9 + i % 3, wide - i), (260 + i, 17 + i // 2)]], rank, iters, monkeypatch)


def test_callers_that_never_finish_in_one_pass_plan_none(monkeypatch):
    from powersgd_b200.paper.reducers import RankKReducer

    monkeypatch.setattr(NativeCompressor, "PANEL_ELEMS", 0)
    send = [torch.randn(600, 1024, device="cuda"), torch.randn(64, 576, device="cuda")]
    reducer = RankKReducer(0, send[0].device, reuse_query=True, rank=2)
    reducer.reduce(send, [torch.empty_like(x) for x in send], [torch.empty_like(x) for x in send])
    assert reducer._native.comp._panel is None
