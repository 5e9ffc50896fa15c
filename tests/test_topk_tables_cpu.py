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


def test_a_call_that_breaks_off_leaves_no_workspace_behind(fake):
    """A call counts in one half of its workspace and clears the other for the next; the halves change places with its last line."""
    halves = []

    def launch(*args):
        halves.append((args[6].value, args[7].value))   # counted in, cleared
        if len(halves) == 3:
            raise KeyboardInterrupt   # as the interpreter raises it behind a foreign call, whose launches have been made
        return 0

    fake.launch, x = launch, torch.randn(100)
    _select(x, None)
    _select(x, None)
    assert halves[1] == halves[0][::-1]
    with pytest.raises(KeyboardInterrupt):
        _select(x, None)
    (broken,) = topk._many_cache.values()
    _select(x, None)   # a workspace of zeros
    (entry,) = topk._many_cache.values()
    assert entry["ws"] is not broken["ws"] and entry["turn"] == 1 and not entry["open"]
