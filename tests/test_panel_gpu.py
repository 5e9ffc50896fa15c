"""The last product and the decompression in one pass over the gradient, against float64 at the edges of its
panels, groups and columns."""
import numpy as np
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD, Config, PowerSGD
from powersgd_b200.cuda_path import NativeCompressor
from powersgd_b200.ops import layout

pytestmark = pytest.mark.gpu

SHAPES = [(5, 23), (70, 27), (64, 576), (129, 650), (33, 1001), (300, 1024), (41, 514), (600, 64), (2500, 24)]


def _draw(gen, shape, off=False):
    """Normal values; `off`: 4 bytes behind a 16-byte boundary, where the kernel takes no gradient."""
    size = torch.Size(shape).numel()
    return torch.randn(size + 4, generator=gen, device="cuda")[1 if off else 0 :][:size].view(shape)


def _tiles_of(nat, name, key):
    """Matrices of a tile list."""
    tiles, count = nat._tiles_dev[name][key]
    return set() if not count else set(np.frombuffer(tiles.cpu().numpy().tobytes()[: count * layout.TILE_DTYPE.itemsize], layout.TILE_DTYPE)["mat"].tolist())


def _check(shapes, rank, iters, monkeypatch, off=(), left=()):
    """The fresh P, the update and the residual from the factors of the launches before. P sums m products in chains of
    at most 12 and a tree of at most 10 additions, less the corrections of r products each; an update sums K
    products: off by at most that many 2^-24 of the terms' sizes (each side rounds to float32). `left`: matrices that
    the launches apart take (`off`: because of where their gradients lie). Their P is a sum in any order, of products of
    values split in two on the tensor cores (2^-20 of a product at most)."""
    monkeypatch.setattr(NativeCompressor, "PANEL_ELEMS", 0)
    gen = torch.Generator(device="cuda").manual_seed(7)
    draw = lambda s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    params = [torch.nn.Parameter(draw(s)) for s in shapes]
    agg = PowerSGD(params, Config(rank=rank, min_compression_rate=0.01, num_iters_per_step=iters, start_compressing_after_num_steps=0))
    for step in range(2 if iters % 2 else 1):   # a step of an odd number that starts on the Q side ends there
        grads = [_draw(gen, s, i in off) for i, s in enumerate(shapes)]
        before = [g.double() for g in grads]
        outs = agg.aggregate(grads)
    core, nat = agg._powersgd, agg._powersgd._native
    torch.cuda.synchronize()
    nat.check()   # no wait inside a kernel ran out
    assert nat._finished and all(agg.is_compressed_mask)
    assert {nat.tiles.mats[mi][2] for key in ("f_rest", "tc_rest") for mi in _tiles_of(nat, "fin", key)} == set(left)
    assert {nat.tiles.mats[mi][2] for key in ("f_rest", "tc_rest") for mi in _tiles_of(nat, "nn", key)} == set(left)
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
            terms = 24 + r + iters if idx not in left else grp.m + 16 + r * iters
            assert ((fresh - (grad @ basis - taken)).abs() <= terms * eps * size).all(), ("P", shapes[idx])
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


@pytest.mark.parametrize("rank,iters", [(1, 2), (4, 2), (8, 1)])
@pytest.mark.parametrize("shape", [(31001, 1024), (31002, 650), (31003, 1001), (250001, 64)])
def test_rings_are_refilled(shape, rank, iters, monkeypatch):
    """At least 13 panels for every group, of four or (64 columns) 16 rows: more than twice what a ring of three to six
    holds, at every access width, with a last panel that is not whole and another matrix behind it."""
    _check([shape, (2001, 700)], rank, iters, monkeypatch)


MIXED = [(260, 5000), (300, 1024), (64, 576), (129, 650), (70, 6300), (513, 300), (33, 1001)]   # 0 and 4 are too wide


@pytest.mark.parametrize("rank,iters", [(1, 2), (2, 2), (4, 2), (8, 1)])
def test_beside_the_launches_apart(rank, iters, monkeypatch):
    """Some matrices are left to the other launches: two whose gradients lie 4 bytes off, and two that are too wide (the
    first, at rank 8, is multiplied by the tensor cores)."""
    _check(MIXED, rank, iters, monkeypatch, off=(1, 5), left=(0, 1, 4, 5))


@pytest.mark.parametrize("rank,iters", [(1, 2), (4, 2), (8, 1)])
def test_overlapped_repeated_and_recorded_launches_leave_the_bits_alone(rank, iters, monkeypatch):
    monkeypatch.setattr(NativeCompressor, "PANEL_ELEMS", 0)

    def run(how):
        gen = torch.Generator(device="cuda").manual_seed(11)
        core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in MIXED], BasicConfig(rank=rank, num_iters_per_step=iters), backend="native")
        grads = [_draw(gen, s, i in (1, 5)) for i, s in enumerate(MIXED)]
        fresh = [_draw(gen, s) for s in MIXED]
        seen = []

        def steps():   # an odd number of half-iterations ends on the Q side in every other step
            for _ in range(1 + iters % 2):
                torch._foreach_add_(grads, fresh)
                outs = core.aggregate(grads)
            return outs

        outs = steps()
        nat = core._native
        assert nat._finished and nat._tiles_dev["fin"]["f_rest"][1] and (rank < 8 or nat._tiles_dev["nn"]["tc_rest"][1])
        if how == "recorded":
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                steps()
        for _ in range(3):
            if how == "recorded":
                graph.replay()
            else:
                if how == "apart":
                    monkeypatch.setattr(nat, "_chained", lambda: False)
                if how != "repeated":
                    nat._tapes.clear()
                outs = steps()
            seen += [x.clone() for x in outs + grads]
        torch.cuda.synchronize()
        nat.check()
        return seen + [core._ps_buffer, core._qs_buffer]

    want = run("apart")
    for how in ("chained", "repeated", "recorded"):
        assert all(torch.equal(a, b) for a, b in zip(run(how), want)), how
