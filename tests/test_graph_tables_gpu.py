"""Descriptor tables built while a CUDA graph is being recorded are put in place once, outside the graph:
its replays must find them intact although the graph's own memory is written over and over."""
import gc
import weakref

import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD, Config, PowerSGD, optimizer_step
from powersgd_b200.cuda_path import capture_scope

pytestmark = pytest.mark.gpu


def test_tables_bound_under_capture_survive_replays():
    shapes = [(96, 200), (300, 260), (64, 27)]
    make = lambda: BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=2, num_iters_per_step=2), backend="native")  # noqa: E731
    g = torch.Generator(device="cuda").manual_seed(0)
    fresh = [torch.randn(s, generator=g, device="cuda") for s in shapes]
    ours, plain = make(), make()
    ours.aggregate([f.clone() for f in fresh])     # builds the native object; its tables are bound anew below
    plain.aggregate([f.clone() for f in fresh])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with capture_scope() as keep, torch.cuda.graph(graph, capture_error_mode="relaxed"):
        for size in (64, 512, 4096, 1 << 16, 1 << 20):   # blocks of every size the tables could be given, written and let go
            scratch = torch.full((size,), -1, dtype=torch.int32, device="cuda")
            del scratch
        grads = [f * 1.0 for f in fresh]
        outs = ours.aggregate(grads)
    assert keep
    for step in range(3):
        for f in fresh:
            f.copy_(torch.randn(f.shape, generator=g, device="cuda"))
        graph.replay()
        want_grads = [f.clone() for f in fresh]
        want = plain.aggregate(want_grads)
        for a, b in zip(list(outs) + grads, list(want) + want_grads):
            assert torch.equal(a, b), step


def test_native_objects_go_with_their_aggregator():
    """No reference cycle keeps pinned memory until the collector runs, which may be during a capture."""
    params = [torch.nn.Parameter(torch.randn(s, device="cuda")) for s in [(96, 200), (33,)]]
    for p in params:
        p.grad = torch.randn_like(p)
    opt = torch.optim.SGD(params, lr=0.1, momentum=0.9)
    agg = PowerSGD(params, Config(rank=2, start_compressing_after_num_steps=0))
    gc.collect()
    gc.disable()
    try:
        for _ in range(3):
            optimizer_step(opt, agg)
        gone = [weakref.ref(agg._powersgd._native), weakref.ref(agg._fused)]
        del agg
        assert all(ref() is None for ref in gone)
    finally:
        gc.enable()


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_tables_can_be_bound_under_every_capture_mode(mode):
    """New tensors bound for the first time inside a recording: the uploads allocate, which a strict recording
    refuses on its own thread."""
    shapes = [(96, 200), (64, 27)]
    make = lambda: BasicPowerSGD([torch.zeros(s, device="cuda") for s in shapes], BasicConfig(rank=2, num_iters_per_step=2), backend="native")  # noqa: E731
    g = torch.Generator(device="cuda").manual_seed(0)
    first, second = ([torch.randn(s, generator=g, device="cuda") for s in shapes] for _ in range(2))
    ours, plain = make(), make()
    before = [f.clone() for f in first]   # stays alive: the recorded call gets tensors at other addresses
    ours.aggregate(before), plain.aggregate([f.clone() for f in first])
    grads, want_grads = ([f.clone() for f in second] for _ in range(2))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with capture_scope() as keep, torch.cuda.graph(graph, capture_error_mode=mode):
        outs = ours.aggregate(grads)
    assert keep
    graph.replay()
    want = plain.aggregate(want_grads)
    for a, b in zip(list(outs) + grads, list(want) + want_grads):
        assert torch.equal(a, b)
