"""The batched selection that writes its output itself: the same bits as the combination of its pairs, call after call
on scratch that one call clears for the next, by lists and the long way, and outputs that lie where others are read."""
import pytest
import torch

from powersgd_b200.ops import topk
from test_topk_gpu import _tensors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("room", [0, 4, topk.CANDIDATES])
@pytest.mark.parametrize("memory", ["other", "none", "own"])
def test_outputs(room, memory, monkeypatch):
    monkeypatch.setattr(topk, "CANDIDATES", room)
    topk._many_cache.clear()
    dev = torch.device("cuda:0")
    tensors, ks = map(list, zip(*_tensors(dev)))
    before = [t.clone() for t in tensors]
    outs = [torch.empty(t.numel() + 1, device=dev)[i % 2 :][: t.numel()] for i, t in enumerate(tensors)]   # every other one 4 bytes off
    mems = {"other": [torch.empty_like(t) for t in tensors], "none": None, "own": tensors}[memory]
    for call in range(3):
        for t, b, o in zip(tensors, before, outs):
            t.copy_(b * (1 + call))
            o.fill_(float("nan"))
        values, positions = topk.topk_abs_many(tensors, ks, mems, outs)
        (entry,) = topk._many_cache.values()
        assert entry["dense"]
        at = 0
        for b, k, o, m in zip(before, ks, outs, mems or [None] * len(ks)):
            v, p = values[at : at + k], positions[at : at + k].long()
            at += k
            x = b * (1 + call)
            assert torch.equal(v.abs().sort(descending=True).values, torch.topk(x.abs(), k).values)
            assert torch.equal(o, torch.zeros_like(x).index_add_(0, p, v))
            assert m is None or torch.equal(m, x.index_fill(0, p, 0.0))
    topk._many_cache.clear()


def test_outputs_where_others_are_read():
    """The output of one tensor is the input of another, or another memory: selected first, combined afterwards."""
    dev = torch.device("cuda:0")
    for clash in ("input", "memory", "output", "length"):
        topk._many_cache.clear()
        g = torch.Generator(device=dev).manual_seed(5)
        x = [torch.randn(30000, generator=g, device=dev) for _ in range(2)]
        before, ks = [t.clone() for t in x], [100, 60]
        mems, outs = [torch.empty_like(t) for t in x], [torch.empty_like(t) for t in x]
        if clash == "input":
            outs[0] = x[1]
        elif clash == "memory":
            outs[1] = mems[0]
        elif clash == "output":
            both = torch.empty(50000, device=dev)
            outs = [both[:30000], both[20000:]]
        else:
            outs[0] = torch.empty(31000, device=dev)
        values, positions = topk.topk_abs_many(x, ks, mems, outs)
        (entry,) = topk._many_cache.values()
        assert not entry["dense"]
        want = [torch.zeros(o.numel(), device=dev).index_add_(0, p.long(), v)
                for o, v, p in zip(outs, values.split(ks), positions.split(ks))]
        if clash != "output":   # (what two of them in one place hold is not defined)
            assert torch.equal(outs[0], want[0]) and torch.equal(outs[1], want[1])
        for b, v, p in zip(before, values.split(ks), positions.split(ks)):
            assert torch.equal(v, b[p.long()])
    topk._many_cache.clear()


def test_another_length_at_the_same_address():
    """A view that is as long as the tensor, then longer and shorter ones that begin where it does, on the tables that the first has left."""
    topk._many_cache.clear()
    g = torch.Generator(device="cuda").manual_seed(6)
    x, room = torch.randn(30000, generator=g, device="cuda"), torch.empty(32000, device="cuda")
    for length in (30000, 31000, 29000, 30000):
        room.fill_(float("nan"))
        values, positions = topk.topk_abs_many([x], [700], None, [room[:length]])
        want, inside = torch.zeros(length, device="cuda"), positions < length
        want.index_add_(0, positions[inside].long(), values[inside])
        assert torch.equal(room[:length], want) and room[length:].isnan().all()
    topk._many_cache.clear()
