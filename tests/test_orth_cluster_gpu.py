"""The orthonormalisation in one launch, a cluster of CTAs per unit, beside the two launches: shares of less than a
row per CTA, whole and ragged shares, rows beyond those a thread keeps, members of a rank-1 group."""
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD
from powersgd_b200.cuda_path import NativeCompressor

pytestmark = pytest.mark.gpu


def _both(shapes, rank, prev, same, collapse=()):
    """(factors before, prev factors, native object, results (basis, copy, cross products) of the two launches and of one)."""
    core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=rank, num_iters_per_step=4), backend="native")
    nat = NativeCompressor(core)
    gen = torch.Generator(device="cuda").manual_seed(sum(shapes[0]) + rank)
    draw = lambda t: t.copy_(torch.randn(t.shape, generator=gen, device="cuda"))  # noqa: E731
    x = draw(core._ps_buffer)
    for view in core._ps:
        for column, of in collapse:
            if column < view.shape[2]:
                view[:, :, column] = 3 * view[:, :, of] if of is not None else 0
    was = x.clone()
    factors = [draw(nat.h_loc[i]) for i in range(prev)]
    if same:
        factors[-1][: x.numel()].copy_(x)
    results = []
    for clusters in (False, True):
        x.copy_(was)
        copy = nat.h_in[3].fill_(float("nan"))
        nat._orth_clusters = {"p": clusters}
        nat.launches = 0
        nat._orth("p", x, copy, factors, nat.cmat[prev], same=same and clusters, clusters=clusters)
        assert nat.launches == (1 if clusters else 2)
        results.append((x.clone(), copy[: x.numel()].clone(), [c.clone() for c in nat.cmat[prev]]))
    return core, factors, results


@pytest.mark.parametrize("rank", [1, 2, 3, 4, 5, 8, 11, 16])
@pytest.mark.parametrize("rows", [1, 5, 31, 32, 33, 1025, 2050, 9001])
@pytest.mark.parametrize("prev,same", [(0, False), (1, True), (2, True), (2, False)])
def test_one_launch_equals_two(rank, rows, prev, same):
    """Both round one float64 solution, whose sums run in another order (relative 1e-13 times the condition, at most some 1e4
    for Gaussian columns), so entries of at most 1 differ by an ulp of 2^-24 at most; cross products, rounded once, by 2^-23 of
    their columns' length. A square factor (rows = rank = 1, rank 5 of 5 rows) is conditioned up to some 1e3: 2^-22."""
    core, factors, (two, one) = _both([(rows, 64), (rows, 64), (33, 50)], rank, prev, same)
    assert torch.equal(one[0], one[1])
    assert (one[0] - two[0]).abs().max() <= 2.0 ** -22
    longest = max([f.norm() for f in factors], default=1.0)
    for a, b in zip(one[2], two[2]):
        assert (a - b).abs().max() <= 2.0 ** -22 * longest


@pytest.mark.parametrize("rank", [2, 4, 8, 16])
@pytest.mark.parametrize("rows", [20, 700, 3000])
def test_collapsed_columns(rank, rows):
    """Zero and dependent columns are replaced alike, from the leading rows as they came in."""
    _core, factors, (two, one) = _both([(rows, 64)], rank, 1, True, collapse=((1, 0), (2, None), (5, 3)))
    assert torch.isfinite(one[0]).all()
    assert (one[0] - two[0]).abs().max() <= 2.0 ** -20
    assert (one[2][0] - two[2][0]).abs().max() <= 2.0 ** -20 * factors[0].norm()


@pytest.mark.parametrize("members", [2, 7, 8, 9, 100])
def test_rank_one_groups(members):
    """One joint norm; cross products member by member, whole members per CTA."""
    _core, factors, (two, one) = _both([(301, 40)] * members, 1, 2, False)
    assert (one[0] - two[0]).abs().max() <= 2.0 ** -22
    for a, b in zip(one[2], two[2]):
        assert (a - b).abs().max() <= 2.0 ** -22 * factors[0].norm()


def test_rule():
    """Small models keep two launches, as do units too long for a cluster and groups with too many members."""
    def rule(shapes, rank, iters=2):
        nat = NativeCompressor(BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=rank, num_iters_per_step=iters), backend="native"))
        return nat._orth_by_rule["p"], nat._orth_by_rule["q"]

    assert rule([(512, 512)], 2) == (True, True)
    assert rule([(512, 511)], 2) == (False, False)
    assert rule([(50257, 2048)], 4) == (False, True)
    assert rule([(4096, 2048)], 8) == (False, True)
    assert rule([(64, 512)] * 700, 1) == (False, False)
    assert rule([(16, 512)] * 700, 1, iters=1) == (True, False)   # 700 x 16 and 700 x 512 rows in one unit
    assert rule([(2048, 2048)], 32) == (False, False)


def test_rule_by_the_number_of_units():
    """More units than run at a time take two launches, but for long ones."""
    def rule(shapes, rank):
        nat = NativeCompressor(BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=rank, num_iters_per_step=2), backend="native"))
        return nat._orth_by_rule["p"], nat._orth_by_rule["q"], nat._orth_clusters["p"]

    for rank in (2, 3, 8, 16):
        assert rule([(128, 512)] * 20, rank) == (True, True, True)
        assert rule([(128, 512)] * 100, rank) == (False, False, False)
    assert rule([(8192, 64)] * 60, 4) == (True, False, True)
    assert rule([(128, 512)] * 100, 1) == (True, False, True)   # one unit, of 12 800 and of 51 200 rows
