"""The launch over the uncompressed tensors starts beside the end of the low-rank launches: bits as when every launch
waits for the one before, for `aggregate`, the optimizer step and the rank-k reducers."""
import pytest
import torch

from powersgd_b200 import Config, PowerSGD, optimizer_step
from powersgd_b200.cuda_path import NativeCompressor

pytestmark = pytest.mark.gpu

# last strips of a launch that fills the GPU several times; vectors of a ragged length, on and off a 16-byte boundary
SHAPES = [(2048, 2304), (1001, 777), (333,), (40000,), (1,), (700, 650)]


def _run(kind, steps=5):
    gen = torch.Generator(device="cuda").manual_seed(1)
    draw = lambda: [torch.randn(s, generator=gen, device="cuda") for s in SHAPES]  # noqa: E731
    seen = []
    if kind in ("rankk", "halfrankk"):
        from powersgd_b200.paper.reducers import HalfRankKReducer, RankKReducer

        red = RankKReducer(3, torch.device("cuda:0"), reuse_query=True, rank=3) if kind == "rankk" else HalfRankKReducer(3, torch.device("cuda:0"), rank=3)
        for _ in range(steps):
            grads, outs, mems = draw(), draw(), draw()
            red.reduce(grads, outs, mems)
            seen += outs + mems[:2] + [mems[5]] + grads
        return seen
    params = [torch.nn.Parameter(p) for p in draw()]
    agg = PowerSGD(params, Config(rank=2, num_iters_per_step=3, start_compressing_after_num_steps=0))
    opt = torch.optim.SGD(params, lr=0.1, momentum=0.9)
    grads = [torch.zeros_like(p) for p in params]
    for p, g in zip(params, grads):
        p.grad = g
    for _ in range(steps):
        torch._foreach_add_(grads, draw())
        if kind == "aggregate":
            seen += [o.clone() for o in agg.aggregate(grads)]
        else:
            optimizer_step(opt, agg)
        seen += [g.clone() for g in grads] + [p.detach().clone() for p in params]
    return seen


@pytest.mark.parametrize("kind", ["aggregate", "step", "rankk", "halfrankk"])
def test_bits_do_not_depend_on_the_overlap(kind, monkeypatch):
    usual = _run(kind)
    monkeypatch.setattr(NativeCompressor, "_chained", lambda self: False)
    apart = _run(kind)
    assert all(torch.equal(a, b) for a, b in zip(usual, apart))
