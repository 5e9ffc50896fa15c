"""The batched selection where its candidate lists suffice, where they do not, and where there are none."""
import pytest
import torch

from powersgd_b200.ops import topk

pytestmark = pytest.mark.gpu


def _tensors(dev):
    g = torch.Generator(device=dev).manual_seed(11)
    normal = lambda n: torch.randn(n, generator=g, device=dev)  # noqa: E731
    flat = normal(70001)
    yield flat[1:], 143                                                                # 4-byte aligned
    yield normal(300000), 614                                                           # some 2 k candidates
    yield torch.rand(200000, generator=g, device=dev), 400                              # an eighth of all are candidates
    yield torch.full((150000,), -0.75, device=dev), 300                                 # all of them
    yield torch.where(torch.rand(90000, generator=g, device=dev) < 0.01, 1.5, 1.0), 1200    # ties at the threshold
    yield normal(9000).sign() * 2.0 ** torch.randint(-126, 120, (9000,), generator=g, device=dev), 77
    yield torch.cat([normal(5000), torch.tensor([float("inf"), -float("inf"), 0.0, -0.0], device=dev)]), 40
    yield torch.zeros(5000, device=dev), 10
    yield normal(1), 1
    yield normal(600), 600


@pytest.mark.parametrize("room", [0, 1, 4])
@pytest.mark.parametrize("memory", ["other", "none", "own"])
def test_selection(room, memory, monkeypatch):
    monkeypatch.setattr(topk, "CANDIDATES", room)
    topk._many_cache.clear()
    dev = torch.device("cuda:0")
    tensors, ks = map(list, zip(*_tensors(dev)))
    before = [t.clone() for t in tensors]
    mems = {"other": [torch.full_like(t, float("nan")) for t in tensors], "none": None, "own": tensors}[memory]
    values, positions = topk.topk_abs_many(tensors, ks, mems)
    topk._many_cache.clear()
    at = 0
    for i, (x, k) in enumerate(zip(before, ks)):
        v, p = values[at : at + k], positions[at : at + k].long()
        at += k
        assert p.unique().numel() == k and torch.equal(v, x[p]), i
        assert torch.equal(v.abs().sort(descending=True).values, torch.topk(x.abs(), k).values), i
        if mems is not None:
            rest = x.clone()
            rest[p] = 0.0
            assert torch.equal(mems[i], rest), i
