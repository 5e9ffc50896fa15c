"""The batched selection where its candidate lists suffice, where they do not, and where there are none."""
import threading

import pytest
import torch

from powersgd_b200.ops import topk

pytestmark = pytest.mark.gpu


def _tensors(dev):
    g = torch.Generator(device=dev).manual_seed(11)
    normal = lambda n: torch.randn(n, generator=g, device=dev)  # noqa: E731
    flat = normal(70001)
    yield flat[1:], 143                                                                # 4-byte aligned
    yield normal(300000), 614                                                           # some 480 candidates
    yield torch.rand(200000, generator=g, device=dev), 400                              # a twentieth of all are candidates
    yield torch.full((150000,), -0.75, device=dev), 300                                 # all of them
    yield torch.where(torch.rand(90000, generator=g, device=dev) < 0.01, 1.5, 1.0), 1200    # ties at the threshold
    yield normal(9000).sign() * 2.0 ** torch.randint(-126, 120, (9000,), generator=g, device=dev), 77
    yield torch.cat([normal(5000), torch.tensor([float("inf"), -float("inf"), 0.0, -0.0], device=dev)]), 40
    yield torch.zeros(5000, device=dev), 10
    yield normal(1), 1
    yield normal(600), 600


@pytest.mark.parametrize("room", [0, 1, 4, topk.CANDIDATES])   # and 403 for the length of the list
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


def test_streams_and_threads_do_not_share_scratch():
    """The same tensors selected from on two streams, by two threads each, while the others are under way."""
    dev = torch.device("cuda:0")
    topk._many_cache.clear()
    tensors, ks = map(list, zip(*_tensors(dev)))
    want = [torch.topk(x.abs(), k).values for x, k in zip(tensors, ks)]
    torch.cuda.synchronize()
    streams, wrong = [torch.cuda.Stream(), torch.cuda.Stream()], []

    def work(stream):
        try:
            with torch.cuda.stream(stream):
                seen = []
                for _ in range(40):
                    values, positions = topk.topk_abs_many(tensors, ks)
                    one, _ = topk.topk_abs(tensors[1], ks[1])
                    seen.append((values, positions, one))
                stream.synchronize()
                for values, positions, one in seen:
                    at = 0
                    for x, k, w in zip(tensors, ks, want):
                        v, p = values[at : at + k], positions[at : at + k].long()
                        at += k
                        if not (torch.equal(v, x[p]) and torch.equal(v.abs().sort(descending=True).values, w)):
                            wrong.append((x.numel(), k))
                    if not torch.equal(one.abs().sort(descending=True).values, want[1]):
                        wrong.append("one tensor")
        except Exception as error:
            wrong.append(error)

    threads = [threading.Thread(target=work, args=(s,)) for s in streams * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:3]
    assert len({entry["ws"].data_ptr() for entry in topk._many_cache.values()}) == 2
    topk._many_cache.clear()


def test_combining_on_two_streams_does_not_share_a_barrier():
    dev = torch.device("cuda:0")
    x = torch.randn(5000, device=dev)
    values, positions = topk.topk_abs(x, 50)
    want = torch.zeros_like(x)
    want[positions.long()] = values
    for stream in (torch.cuda.Stream(), torch.cuda.Stream()):   # one after the other
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            out = torch.full_like(x, 7.0)
            topk.sparse_combine(values.view(1, -1), positions.view(1, -1), [out], [50], 1.0)
        torch.cuda.synchronize()
        assert torch.equal(out, want) and topk._combine_scratch[dev, stream.cuda_stream][1].item() == 0
    assert topk.sparse_combine_status(dev) == 0


@pytest.mark.parametrize("beyond", [0, 1, 100_000])
def test_a_list_longer_than_one_block_walks_goes_the_long_way(beyond):
    """Entries in the threshold's eighth of an octave: as many as the list of a tensor of 1 M entries holds, or more."""
    dev = torch.device("cuda:0")
    topk._many_cache.clear()
    g = torch.Generator(device=dev).manual_seed(3)
    n, room = 1 << 20, topk.CANDIDATES + 512
    x = torch.rand(n, generator=g, device=dev) * 0.5
    at = torch.randperm(n, generator=g, device=dev)[: room + beyond]
    x[at] = 1.0 + 0.124 * torch.rand(len(at), generator=g, device=dev)
    memory = torch.full_like(x, 7.0)
    values, positions = topk.topk_abs_many([x], [2000], [memory])
    p = positions.long()
    assert torch.equal(values.sort(descending=True).values, torch.topk(x, 2000).values) and torch.equal(values, x[p])
    assert torch.equal(memory, x.index_fill(0, p, 0.0))
    (entry,) = topk._many_cache.values()
    listed = int(entry["ws"][2048 + 2048 + 512 + 2])
    assert entry["cand_v"].numel() == room and listed == (0 if beyond else room)
    topk._many_cache.clear()
