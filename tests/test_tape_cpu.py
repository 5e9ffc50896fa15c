"""When launches are repeated from the library's record, and when they are not (host code only, a library that launches nothing)."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from powersgd_b200 import cuda_path
from powersgd_b200.cuda_path import NativeFlatAllReduce


class _Lib:
    """Counts the launches; `written` of each get onto the record."""

    def __init__(self, written):
        self.written, self.made, self.repeated = written, 0, 0

    def psgd_tape_begin(self):
        self.made_before = self.made
        return 1

    def psgd_tape_end(self):
        return self.written * (self.made - self.made_before)

    def psgd_tape_free(self, tape):
        pass

    def psgd_tape_replay(self, tape, stream):
        self.repeated += 1
        return 0

    def psgd_flat_launch(self, *args):
        self.made += 1
        return 0


@pytest.mark.parametrize("written", [0, 1])
def test_a_flat_launch_is_repeated_only_if_it_was_written_down(written, monkeypatch):
    monkeypatch.setattr(cuda_path, "_stream_ptr", lambda: ctypes.c_void_p(0))
    flat = object.__new__(NativeFlatAllReduce)
    buf = torch.zeros(4)
    flat.lib, flat.path, flat.launches, flat.comm, flat.n_pad, flat._tapes = _Lib(written), "local", 0, None, 0, {}
    flat._keep_inputs, flat._vec, flat._nblocks, flat._flat = False, 1, 1, None
    flat._items_dev = flat._block_item = flat._block_first = buf
    for _ in range(3):
        flat._run(buf, 1, sgd=True)
    assert (flat.lib.made, flat.lib.repeated) == ((1, 2) if written else (3, 0))
    assert flat.launches == 3
