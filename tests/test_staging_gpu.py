"""The factor values that the CUDA-core products stage: every width of access and copy, ranks at and below the template
rank, ragged last chunks, factors that begin off a 16-byte boundary."""
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rank", [1, 2, 3, 4, 7, 8, 16, 32])
@pytest.mark.parametrize("lead", [(), ((5, 7),)])   # the second shifts the factors of those behind by 25 and 35 floats
def test_products_against_float64(rank, lead, monkeypatch):
    """Both products of a step of two half-iterations from the factors the launches used. A sum of n products in any order is off by
    at most n 2^-24 of the sum of their sizes, the correction of the second by as much of its terms."""
    monkeypatch.setenv("PSGD_B200_GEMM", "ffma")
    shapes = list(lead) + [(33, 129), (300, 1), (257, 1025), (64, 2050), (130, 650), (31, 127), (260, 128), (1030, 40)]
    g = torch.Generator(device="cuda").manual_seed(rank)
    grads = [torch.randn(s, generator=g, device="cuda") for s in shapes]
    before = [x.double() for x in grads]
    core = BasicPowerSGD([torch.zeros_like(x) for x in grads], BasicConfig(rank=rank, num_iters_per_step=2), backend="native")
    core.aggregate(grads)
    nat = core._native
    assert not nat.uses_tensor_cores
    for grp in core.plan.groups:
        for pos, idx in enumerate(grp.members):
            m, r = before[idx], grp.r
            p = lambda buf: buf[grp.p_offset + pos * grp.n * r :][: grp.n * r].view(grp.n, r).double()  # noqa: E731
            q = lambda buf: buf[grp.q_offset + pos * grp.m * r :][: grp.m * r].view(grp.m, r).double()  # noqa: E731
            left, right, basis = p(nat.h_in[0]), q(nat.h_loc[0]), q(nat.h_in[1])
            assert ((right - m.T @ left).abs() <= grp.n * 2.0 ** -24 * (m.abs().T @ left.abs()) + 1e-30).all(), (shapes[idx], "M^T P")
            taken, size = left @ (right.T @ basis), left.abs() @ (right.abs().T @ basis.abs())
            bound = (grp.m + 2 * r) * 2.0 ** -24 * (m.abs() @ basis.abs() + size)
            assert ((p(nat.h_loc[1]) - (m @ basis - taken)).abs() <= bound + 1e-30).all(), (shapes[idx], "M Q")


@pytest.mark.parametrize("rank", [1, 2, 3, 4, 8])
def test_product_of_more_tiles_than_run_at_a_time(rank, monkeypatch):
    """M Q of a tall matrix: some 470 tiles of 32 rows, which all copy the same rows of Q-hat."""
    monkeypatch.setenv("PSGD_B200_GEMM", "ffma")
    g = torch.Generator(device="cuda").manual_seed(rank)
    m = torch.randn(15001, 132, generator=g, device="cuda")
    core = BasicPowerSGD([torch.zeros_like(m)], BasicConfig(rank=rank, num_iters_per_step=1), backend="native")
    core.aggregate([m.clone()])             # left factor first ...
    core.aggregate([m.clone()])             # ... right factor now: one M Q
    nat = core._native
    assert len(nat._tile_arrays["nn"]["f"]) > 3 * 148
    q = nat.h_in[0][: 132 * rank].view(132, rank).double()
    p = nat.h_loc[0][: 15001 * rank].view(15001, rank).double()
    m = m.double()
    assert ((p - m @ q).abs() <= 132 * 2.0 ** -24 * (m.abs() @ q.abs()) + 1e-30).all()
