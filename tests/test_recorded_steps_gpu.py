"""Steps recorded in a CUDA graph by the program itself (`torch.cuda.graph` around `optimizer_step`): what
happens between the recording and its replays - other learning rates, other tensors - must reach the
replays exactly as it reaches eager steps, and must never pull memory away from under them."""
import gc
import time
import weakref

import pytest
import torch

from powersgd_b200 import Config, PowerSGD, optimizer_step
from powersgd_b200.cuda_path import capture_scope
from powersgd_b200.ops.recording import release_finished

pytestmark = pytest.mark.gpu

SHAPES = [(128, 300), (70, 129), (33,)]


def _tensors(shapes, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(s, generator=g, device="cuda") for s in shapes]


class _Program:
    """A model's tensors, SGD with momentum, and a step that accumulates the same fresh gradients each time."""

    def __init__(self, dampening=0.0):
        self.params = [torch.nn.Parameter(x) for x in _tensors(SHAPES, 9)]
        for p, x in zip(self.params, _tensors(SHAPES, 10)):
            p.grad = x
        self.optimizer = torch.optim.SGD(self.params, lr=0.1, momentum=0.9, dampening=dampening)
        # two half-iterations per step: every step starts on the same side, so one graph serves them all
        self.aggregator = PowerSGD(self.params, Config(rank=2, num_iters_per_step=2, start_compressing_after_num_steps=0))
        self.fresh = _tensors(SHAPES, 11)

    def step(self, rate=None):
        if rate is not None:
            self.optimizer.param_groups[0]["lr"] = rate
        torch._foreach_add_([p.grad for p in self.params], self.fresh)
        optimizer_step(self.optimizer, self.aggregator)

    def record(self, *rates):
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for rate in rates:
                self.step(rate)
        return graph

    def state(self):
        torch.cuda.synchronize()
        moms = [self.optimizer.state[p]["momentum_buffer"] for p in self.params]
        return [t.clone() for p, m in zip(self.params, moms) for t in (p.detach(), p.grad, m)]


def _same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a.state(), b.state()))


@pytest.mark.parametrize("dampening", [0.0, 0.3])
def test_replays_use_the_rate_of_the_last_prepared_step(dampening):
    """A fresh optimizer, one eager step, the second step recorded; then more changes of the rate than the
    table's ring has slots, eager steps and replays in turn."""
    recorded, eager = _Program(dampening), _Program(dampening)
    recorded.step(), eager.step()
    if dampening:   # the first step's buffers take the whole gradient, the steps from here on do not
        recorded.step(), eager.step()
    graph = recorded.record(None)
    rates = [0.05, 0.02, 0.2, 0.01, 0.3, 0.07, 0.15]
    for i, rate in enumerate(rates):
        recorded.step(rate), eager.step(rate)
        for _ in range(2 if i == 0 else 1):
            graph.replay()
            eager.step()
        assert _same(recorded, eager), i


def test_rate_changed_for_the_recorded_step_itself():
    recorded, eager = _Program(), _Program()
    recorded.step(), eager.step()
    graph = recorded.record(0.03)
    for _ in range(2):
        graph.replay()
        eager.step(0.03)
    assert _same(recorded, eager)
    recorded.step(0.2), eager.step(0.2)
    graph.replay()   # follows the eager step
    eager.step()
    assert _same(recorded, eager)


def test_two_steps_of_one_recording_with_rates_of_their_own():
    recorded, eager = _Program(), _Program()
    recorded.step(), eager.step()
    graph = recorded.record(0.03, 0.4)
    for _ in range(3):
        graph.replay()
        eager.step(0.03), eager.step(0.4)
    assert _same(recorded, eager)


def test_first_step_recorded_on_the_stream_of_the_eager_ones():
    """Recorded without waiting for the eager step before it, on the same stream: that step may still be
    running and keeps its rate, the recorded one has its own."""
    recorded, eager = _Program(), _Program()
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        recorded.step(), recorded.step()
        graph.capture_begin()
        recorded.step(0.03)
        graph.capture_end()
        graph.replay()
    torch.cuda.current_stream().wait_stream(stream)
    for rate in (None, None, 0.03):
        eager.step(rate)
    assert _same(recorded, eager)


def _write_over_free_memory():
    """Blocks of every size the tables and the scratch of a step could have had, several of each, written."""
    return [torch.full((size,), -1, dtype=torch.int32, device="cuda") for size in (8, 64, 128, 512, 2048, 8192, 1 << 15, 1 << 17) for _ in range(24)]


def _step_on_other_gradients(program):
    own = [p.grad for p in program.params]
    other = _tensors(SHAPES, 77)
    for p, x in zip(program.params, other):
        p.grad = x
    program.step()
    for p, x in zip(program.params, own):
        p.grad = x
    return other


def test_replay_after_other_tensors_were_bound():
    """An eager step on other gradient tensors replaces the descriptor tables and the scratch; the graph
    still refers to the old ones."""
    recorded, eager = _Program(), _Program()
    recorded.step(), eager.step()
    graph = recorded.record(None)
    others = _step_on_other_gradients(recorded), _step_on_other_gradients(eager)
    junk = _write_over_free_memory()
    for _ in range(2):
        graph.replay()
        eager.step()
    assert _same(recorded, eager)
    assert all(torch.equal(a, b) for a, b in zip(*others))
    assert all(bool((j == -1).all()) for j in junk)


def _refs(native):
    return [weakref.ref(t) for t in (native._tickets, native._partial, native._mats_dev)]


def test_what_was_recorded_goes_with_the_aggregator():
    """Other tensors bound again and again keep nothing; a recording keeps what it refers to, once, until
    the aggregator goes."""
    recorded = _Program()
    recorded.step()
    unrecorded = _refs(recorded.aggregator._powersgd._native)
    _step_on_other_gradients(recorded)
    assert all(ref() is None for ref in unrecorded)
    recorded.step()
    refs = _refs(recorded.aggregator._powersgd._native)
    graphs = [recorded.record(None) for _ in range(3)]
    count = len(recorded.aggregator._powersgd._native._kept)
    graphs.append(recorded.record(None))
    assert len(recorded.aggregator._powersgd._native._kept) == count
    _step_on_other_gradients(recorded)
    assert all(ref() is not None for ref in refs)
    del graphs, recorded
    gc.collect()
    assert all(ref() is None for ref in refs)


def test_a_scope_has_what_was_recorded():
    recorded = _Program()
    recorded.step()
    refs = _refs(recorded.aggregator._powersgd._native)
    with capture_scope() as keep:
        graph = recorded.record(None)
    _step_on_other_gradients(recorded)
    assert all(ref() is not None for ref in refs)
    del graph, keep
    assert all(ref() is None for ref in refs)


def test_what_a_graph_alone_refers_to_goes_with_it():
    """Functions without an object of their own (the top-k tables) leave it to the graph."""
    from powersgd_b200.ops import recording
    from powersgd_b200.ops.topk import topk_abs_many

    x = torch.randn(4096, device="cuda")
    topk_abs_many([x], [16])
    before = set(recording._kept)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        topk_abs_many([x], [16])
    mine = set(recording._kept) - before
    release_finished()
    assert mine and mine <= set(recording._kept)
    del graph
    gc.collect()
    torch.cuda.synchronize()
    until = time.monotonic() + 20   # the graph says so on a thread of the driver
    while mine & set(recording._kept) and time.monotonic() < until:
        release_finished()
        time.sleep(0.01)
    assert not mine & set(recording._kept)


@pytest.mark.parametrize("reducer", ["TopKReducer", "GlobalTopKReducer"])
@pytest.mark.parametrize("warm", [False, True])
def test_recorded_topk_reduce_survives_other_tensor_sets(reducer, warm):
    """The reducers keep tables for the last few sets of tensors; a recorded call must not depend on them."""
    from powersgd_b200.paper import reducers

    shapes = [(300, 200), (64, 27), (129,), (1,)]
    red = getattr(reducers, reducer)(0, torch.device("cuda:0"), compression=1 / 16)
    new = lambda seed: (_tensors(shapes, seed), [torch.full(s, 7.0, device="cuda") for s in shapes], [torch.full(s, 7.0, device="cuda") for s in shapes])  # noqa: E731
    send, out, memory = new(0)
    if warm:
        red.reduce(send, out, memory)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        red.reduce(send, out, memory)
    held = [new(seed) for seed in range(1, 7)]
    for other in held:
        red.reduce(*other)
    junk = _write_over_free_memory()
    for seed in (20, 21):
        for x, fresh in zip(send, _tensors(shapes, seed)):
            x.copy_(fresh)
        graph.replay()
        want = new(seed)
        red.reduce(*want)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out + memory, want[1] + want[2]))
    assert all(bool((j == -1).all()) for j in junk)


def test_train_step_uses_a_loaded_optimizer_state():
    """The graph of a TrainStep updates the buffers that were there when it was recorded; after
    `optimizer.load_state_dict` there are others."""
    import copy

    from powersgd_b200.engine import TrainStep
    from powersgd_b200.models.mlp import MLP

    x, y = torch.randn(32, 64, device="cuda"), torch.randint(0, 10, (32,), device="cuda")

    def run(cuda_graph):
        torch.manual_seed(0)
        model = MLP(64, 128, 10).cuda()
        opt = torch.optim.SGD(model.parameters(), lr=0.05, momentum=0.9)
        agg = PowerSGD(list(model.parameters()), Config(rank=1, num_iters_per_step=1, start_compressing_after_num_steps=0))
        step = TrainStep(model, torch.nn.functional.cross_entropy, opt, agg, cuda_graph=cuda_graph)
        saved, losses = None, []
        for i in range(12):
            if i == 3:
                saved = copy.deepcopy(opt.state_dict())
            if i in (7, 10):
                opt.load_state_dict(saved)
            losses.append(step(x, y).clone())
        assert bool(step._graphs) == cuda_graph
        torch.cuda.synchronize()
        return losses + [t.detach().clone() for p in model.parameters() for t in (p, opt.state[p]["momentum_buffer"])]

    for a, b in zip(run(True), run(False)):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-6)   # the library may choose other kernels under capture
