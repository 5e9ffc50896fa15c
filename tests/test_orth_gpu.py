"""The orthonormalisation launches against float64: ragged chunks, units of many chunks, ranks below and
at the template rank, collapsed columns, the joint norm of a rank-1 group, and the cross products."""
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD

pytestmark = pytest.mark.gpu


def _compressor(shapes, rank):
    dev = torch.device("cuda:0")
    core = BasicPowerSGD([torch.zeros(s, device=dev) for s in shapes], BasicConfig(rank=rank, num_iters_per_step=3), backend="native")
    core.aggregate([torch.randn(s, device=dev) for s in shapes])   # builds and binds the native object
    return core, core._native


@pytest.mark.parametrize("rank", [1, 2, 3, 4, 7, 8, 11, 16, 20, 32])
@pytest.mark.parametrize("rows", [40, 511, 513, 2049, 21001])
def test_basis_and_cross_products(rank, rows):
    """Two equal matrices and a short one; two earlier factors. The basis is rounded to float32 once
    (2^-24 per entry of unit columns), so Q^T Q is off by at most about 2 r 2^-24 entry by entry, and the
    cross products, rounded once too, by 2^-24 of |f| plus what the rounding of Q adds: r |f| 2^-24."""
    core, nat = _compressor([(rows, 64), (rows, 64), (33, 50)], rank)
    g = torch.Generator(device="cuda").manual_seed(rows + rank)
    draw = lambda t: t.copy_(torch.randn(t.shape, generator=g, device="cuda"))  # noqa: E731
    x = draw(core._ps_buffer)
    before = [v.double().clone() for v in core._ps]
    prev = [draw(nat.h_loc[0]), draw(nat.h_loc[1])]
    copy = nat.h_in[2].fill_(float("nan"))
    nat._orth("p", x, copy, prev, nat.cmat[2])
    assert torch.equal(copy[: x.numel()], x)
    mat = 0
    for view, was, grp in zip(core._ps, before, core.plan.groups):
        r = grp.r
        norm = was.norm()
        for b in range(grp.batch):
            q = view[b].double()
            if r == 1:   # one norm for the whole group
                assert (q - was[b] / norm).abs().max() <= 2.0 ** -22
            else:
                assert (q.T @ q - torch.eye(r, device="cuda")).abs().max() <= 2 * r * 2.0 ** -23
                basis = torch.linalg.qr(was[b])[0]
                assert (q - basis @ (basis.T @ q)).norm() <= r * 2.0 ** -22 * 8
            for p, c in zip(prev, nat.cmat[2]):
                f = p[grp.p_offset + b * grp.n * r : grp.p_offset + (b + 1) * grp.n * r].view(grp.n, r).double()
                got = c[mat * 1024 : mat * 1024 + r * r].view(r, r).double()
                assert (got - f.T @ q).abs().max() <= 4 * r * 2.0 ** -24 * f.norm(dim=0).max()
            mat += 1


@pytest.mark.parametrize("rank", [2, 4, 8, 16])
@pytest.mark.parametrize("rows", [20, 700, 5000])
def test_collapsed_columns_are_replaced(rank, rows):
    """Zero, repeated and tiny dependent columns: the result is orthonormal all the same, and the columns
    that were fine still span what they spanned."""
    core, nat = _compressor([(rows, 64)], rank)
    g = torch.Generator(device="cuda").manual_seed(rank)
    x = core._ps[0][0]
    x.copy_(torch.randn(x.shape, generator=g, device="cuda"))
    x[:, 1] = x[:, 0] * 3
    if rank > 2:
        x[:, 2] = 0
    if rank > 4:
        x[:, 5] = x[:, 3] - x[:, 4]
    was = x.double().clone()
    nat._orth("p", core._ps_buffer, nat.h_in[0], [], [])
    q = x.double()
    assert torch.isfinite(q).all()
    assert (q.T @ q - torch.eye(rank, device="cuda")).abs().max() <= 2 * rank * 2.0 ** -23
    alive = [c for c in range(rank) if c not in (1, 2, 5)]
    kept = was[:, alive]
    assert (kept - q @ (q.T @ kept)).norm() <= 1e-6 * kept.norm()


def test_long_unit_has_a_bounded_number_of_chunks():
    """Every chunk reads the partial sums of all chunks of its unit, so their number may not grow with its
    length. Chunks keep to one member of a rank-1 group: there it grows with the members, and only with them."""
    for rank, most in ((1, 256), (4, 256), (8, 128), (16, 80), (32, 48)):
        for rows in (1, 512, 513, 50257, 1_000_003):
            core = BasicPowerSGD([torch.zeros(rows, 40, device="cuda")], BasicConfig(rank=rank), backend="native")
            from powersgd_b200.cuda_path import NativeCompressor

            nat = NativeCompressor(core)
            assert 1 <= nat.n_chunks["p"] <= most
    for members in (2, 300, 700):
        core = BasicPowerSGD([torch.zeros(64, 40, device="cuda")] * members, BasicConfig(rank=1), backend="native")
        assert NativeCompressor(core).n_chunks["p"] == members
    core = BasicPowerSGD([torch.zeros(5000, 40, device="cuda")] * 300, BasicConfig(rank=1), backend="native")
    assert NativeCompressor(core).n_chunks["p"] <= 2 * 300


def test_rank_one_group_of_many_members():
    """More members than a long unit may have chunks: one joint norm, and cross products member by member,
    under the bounds of the test above."""
    members, rows = 700, 64
    core, nat = _compressor([(rows, 40)] * members, 1)
    g = torch.Generator(device="cuda").manual_seed(1)
    draw = lambda t: t.copy_(torch.randn(t.shape, generator=g, device="cuda"))  # noqa: E731
    x = draw(core._ps_buffer)
    was, prev = core._ps[0].double().clone(), [draw(nat.h_loc[0]), draw(nat.h_loc[1])]
    nat._orth("p", x, nat.h_in[2], prev, nat.cmat[2])
    q = core._ps[0].double()
    assert (q - was / was.norm()).abs().max() <= 2.0 ** -22
    for p, c in zip(prev, nat.cmat[2]):
        f = p[: members * rows].view(members, rows).double()
        got = c.view(-1, 1024)[:members, 0].double()
        assert (got - (f * q.view(members, rows)).sum(1)).abs().max() <= 4 * 2.0 ** -24 * f.norm(dim=1).max()
