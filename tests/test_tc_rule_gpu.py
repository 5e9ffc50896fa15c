"""Which lists take the tensor cores, and both ways beside each other where the rule changes hands."""
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD

pytestmark = pytest.mark.gpu


def _core(shapes, rank, iters=2):
    core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=rank, num_iters_per_step=iters), backend="native")
    g = torch.Generator(device="cuda").manual_seed(rank)
    grads = [torch.randn(s, generator=g, device="cuda") for s in shapes]
    out = core.aggregate(grads)
    return core, [o.clone() for o in out] + grads


@pytest.mark.parametrize("shapes,rank,tc", [([(512, 512)] * 4, 8, False), ([(1024, 1024)] * 8, 8, False), ([(1024, 1025)] * 8, 8, False),
                                            ([(1024, 1028)] * 8, 8, True), ([(1024, 1024)] * 4, 16, False), ([(1024, 1028)] * 4, 11, True),
                                            ([(2052, 512)], 8, True), ([(512, 4100)], 8, True), ([(2048, 4096)], 8, False), ([(512, 512)] * 4, 17, True), ([(512, 512)] * 4, 7, False)])
def test_rule(shapes, rank, tc):
    assert _core(shapes, rank)[0]._native.uses_tensor_cores == tc


@pytest.mark.parametrize("rank,iters", [(8, 1), (8, 2), (11, 3), (16, 2)])
def test_both_ways_agree(rank, iters, monkeypatch):
    """Gaussian matrices, whose leading directions are of nearly equal size: a product's relative error (some 1e-6 on the tensor cores)
    turns the basis by about 30 times that at most, and what is subtracted with it."""
    shapes = [(512, 640), (512, 640), (1000, 516)]
    _, here = _core(shapes, rank, iters)
    monkeypatch.setenv("PSGD_B200_GEMM", "tc")
    core, there = _core(shapes, rank, iters)
    assert core._native.uses_tensor_cores
    for a, b in zip(here, there):
        assert ((a - b).norm() / b.norm()).item() < 1e-4
