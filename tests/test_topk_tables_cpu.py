"""What the batched selection keeps from one call for the next (host code only, a library that launches nothing)."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from powersgd_b200.ops import topk


@pytest.fixture
def fake(monkeypatch):
    """Stands for the native library: `fake.launch(...)` is called with what a launch gets."""
    lib = SimpleNamespace(psgd_topk_item_bytes=lambda: 64, psgd_topk_workspace_ints=lambda: 8)
    lib.launch = lambda *args: 0
    lib.psgd_topk_abs_many = lambda *args: lib.launch(*args)
    monkeypatch.setattr(topk.native, "lib", lambda: lib)
    monkeypatch.setattr(topk, "_current_stream", lambda: ctypes.c_void_p(0))
    monkeypatch.setattr(topk, "_many_cache", {})
    for name in ("is_recorded", "release_finished"):
        monkeypatch.setattr(topk, name, lambda *args: False)
    monkeypatch.setattr(topk, "outside_capture", lambda device: torch.no_grad())
    return lib


def _select(x, outs):
    return topk._select([x], [5], [None], outs, torch.empty(5), torch.empty(5, dtype=torch.int32))


def test_an_output_of_another_length_at_the_same_address(fake):
    """Written by the selection only where it is as long as the tensor, whatever an earlier call brought to that address."""
    x, room = torch.randn(100), torch.empty(120)
    assert _select(x, [room[:100]])
    assert not _select(x, [room[:90]])
    assert not _select(x, [room])
    assert _select(x, [room[:100]])
    assert not _select(x, None)
