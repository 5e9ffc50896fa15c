"""The phases that a reducer of one worker reports to its timer, whatever its launches are fused into (host code only)."""
from contextlib import contextmanager

import pytest
import torch

from powersgd_b200.paper import reducers as R


class _Phases:
    def __init__(self):
        self.entered, self.now = [], []

    @contextmanager
    def __call__(self, label, epoch=-1.0, verbosity=1):
        self.entered.append(label)
        self.now.append(label)
        yield
        self.now.pop()


def test_top_k_reports_gathering_and_combining():
    timer, out, mem = _Phases(), [torch.empty(40)], [torch.empty(40)]
    R.TopKReducer(1, "cpu", timer, compression=0.25).reduce([torch.randn(40)], out, mem)
    assert timer.entered == ["reduce.flatpack", "reduce.topk", "reduce.gather", "reduce.combine"]


@pytest.mark.parametrize("kind", [R.RankKReducer, R.HalfRankKReducer])
def test_rank_k_times_the_vectors(kind, monkeypatch):
    timer, calls = _Phases(), []

    class Driver:
        launches, core = 0, None

        def rank_k(self, matrices):
            calls.append(("matrices", timer.now[-1]))

        def half_rank_k(self, matrices, compute_p):
            self.rank_k(matrices)

        def reduce_vectors(self, vectors, early=False):
            calls.append(("vectors", timer.now[-1]))

    red = kind(1, "cpu", timer, rank=2)
    red.reuse_query = True
    red.p_memory = red.q_memory = torch.zeros(4)
    monkeypatch.setattr(red, "_native_driver", lambda matrices, iters: (Driver(), False))
    vector, matrix = [(torch.zeros(5),) * 3], [(torch.zeros(4, 4),) * 3]
    red._reduce_native(vector, matrix)
    assert sorted(calls) == [("matrices", "reduce.lowrank"), ("vectors", "reduce.rank1")]


@pytest.mark.parametrize("kind", [R.RankKReducer, R.HalfRankKReducer])
def test_rank_k_takes_iterators(kind):
    """The lists are walked once."""
    def reduced(wrap):
        g = torch.Generator().manual_seed(3)
        grads = [torch.randn(s, generator=g) for s in ((8, 6), (5,), (3, 4, 2))]
        outs, mems = [torch.zeros_like(x) for x in grads], [torch.zeros_like(x) for x in grads]
        bits = kind(7, "cpu", _Phases(), rank=2).reduce(wrap(grads), wrap(outs), wrap(mems))
        return bits, outs + mems

    (bits, listed), (walked_bits, walked) = reduced(list), reduced(iter)
    assert bits == walked_bits and all(torch.equal(a, b) for a, b in zip(listed, walked))
