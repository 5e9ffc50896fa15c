"""Checks of whole lists of tensors: the extension and the Python form answer alike."""
import pytest
import torch

from powersgd_b200.ops import scan

native = pytest.mark.skipif(scan._native is None, reason="extension not built")


class Sub(torch.Tensor):
    pass


def _lists():
    w = torch.randn(4, 3, 2, 2)
    yield [w, w.to(memory_format=torch.channels_last), torch.zeros(0), torch.ones(1, 5, 1, 1)]
    yield (torch.randn(3, 4).t(), torch.nn.Parameter(torch.randn(5)))
    yield [torch.randn(6)[1:], torch.randn(4, 6)[:, :3]]
    yield [torch.randn(2).as_subclass(Sub), torch.randn(2)]
    yield [torch.randn(2).double(), torch.zeros(2, dtype=torch.int32)]
    yield []


@native
@pytest.mark.parametrize("i", range(6))
def test_lists(i, monkeypatch):
    tensors = list(_lists())[i]
    with_none = list(tensors) + [None]
    ask = lambda: (scan.addresses(tensors), scan.addresses(with_none), scan.addresses(None), scan.sizes(tensors), scan.usable(tensors), scan.usable(tensors, True))  # noqa: E731
    here = ask()
    monkeypatch.setattr(scan, "_native", None)
    assert here == ask()


@native
def test_unknown_objects_are_left_to_python():
    known = scan._native
    assert known.addresses([torch.randn(2).as_subclass(Sub)]) is None and known.sizes(iter([])) is None and known.addresses([1]) is None
    assert torch.func.vmap(lambda x: torch.tensor(known.addresses([x]) is None))(torch.randn(3, 2)).all()
    assert known.usable([torch.randn(2).to_sparse()], 0) is None
    assert known.grad_addresses([torch.nn.Parameter(torch.randn(2))]) is None


def _change(what, params, opt):
    if what == "no gradient":
        params[1].grad = None
    elif what == "transposed gradient":
        params[0].grad = torch.randn(3, 4).t()
    elif what == "channels last":
        params[3].data = params[3].data.to(memory_format=torch.channels_last)
        params[3].grad = params[3].grad.to(memory_format=torch.channels_last)
    elif what == "channels last gradient":
        params[3].grad = params[3].grad.to(memory_format=torch.channels_last)
    elif what == "double":
        params[0].data = params[0].data.double()
    elif what == "strided parameter":
        params[0].data = torch.randn(8, 6)[::2, ::2]
    elif what == "some buffers":
        opt.state[params[0]]["momentum_buffer"] = torch.zeros(4, 3)
    elif what in ("all buffers", "buffer layout"):
        for p in params:
            opt.state[p]["momentum_buffer"] = torch.zeros_like(p)
        if what == "buffer layout":
            opt.state[params[0]]["momentum_buffer"] = torch.zeros(3, 4).t()
    elif what == "empty state":
        opt.state[params[0]]["momentum_buffer"] = None
    elif what in ("maximize", "differentiable"):
        opt.param_groups[1][what] = True
    elif what == "subclass":
        params[1].grad = torch.randn(5).as_subclass(Sub)


CHANGES = ["nothing", "no gradient", "transposed gradient", "channels last", "channels last gradient", "double", "strided parameter",
           "some buffers", "all buffers", "buffer layout", "empty state", "maximize", "differentiable", "subclass"]


@native
@pytest.mark.parametrize("what", CHANGES)
def test_optimizers(what, monkeypatch):
    params = [torch.nn.Parameter(torch.randn(s)) for s in [(4, 3), (5,), (1, 7), (6, 3, 2, 2)]]
    for p in params:
        p.grad = torch.randn(p.shape)
    opt = torch.optim.SGD([{"params": params[:2]}, {"params": params[2:]}], lr=0.1, momentum=0.9)
    _change(what, params, opt)
    here, keys = scan.step_fits(opt), None if what == "no gradient" else scan.grad_addresses(params)
    assert here == (what in ("nothing", "channels last", "all buffers", "empty state", "subclass"))
    monkeypatch.setattr(scan, "_native", None)
    assert here == scan.step_fits(opt)
    assert keys is None or keys == scan.grad_addresses(params)


@pytest.mark.parametrize("target,taken", [("scan_target()", True), ("scan_target() + '0'", False), ("'torch 2.6.0, python 3.11.0'", False), (None, False)])
def test_an_extension_for_another_pytorch_is_left_alone(target, taken, tmp_path):
    path = tmp_path / "_tensor_scan.py"
    path.write_text("from powersgd_b200.csrc.build import scan_target\n" + (f"target = {target}\n" if target else ""))
    assert (scan._load(str(path)) is not None) == taken


@native
def test_the_extension_of_this_tree_says_what_it_was_compiled_for():
    assert scan._load(str(scan.SCAN_LIB)).target == scan.scan_target()
