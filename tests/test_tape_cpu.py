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


MEMORY = r"""
#include <stdlib.h>
#include <new>
bool full = false;
void* operator new(size_t n) {
  void* p = full ? nullptr : malloc(n);
  if (p == nullptr) throw std::bad_alloc();
  return p;
}
void* operator new[](size_t n) { return operator new(n); }
void operator delete(void* p) noexcept { free(p); }
void operator delete[](void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
void operator delete[](void* p, size_t) noexcept { free(p); }
"""
HARNESS = r"""
#include "psgd_host.cpp"
extern bool full;
int main() {
  const long long value = 7;
  const void* args[] = {&value};
  const size_t sizes[] = {sizeof(value)};
  void* tape = psgd_tape_begin();
  psgd_tape_add(nullptr, 1, 32, 0, 0, 1, 1, args, sizes);
  psgd_tape_add(nullptr, 1, 32, 0, 0, 1, 1, args, sizes);
  if (psgd_tape_end() != 2) return 1;
  psgd_tape_free(tape);
  tape = psgd_tape_begin();
  psgd_tape_add(nullptr, 1, 32, 0, 0, 1, 1, args, sizes);
  full = true;
  psgd_tape_add(nullptr, 1, 32, 0, 0, 1, 1, args, sizes);
  full = false;
  if (psgd_tape_end() != -1) return 2;
  psgd_tape_free(tape);
  full = true;
  tape = psgd_tape_begin();
  const int count = psgd_tape_end();
  full = false;
  if (tape != nullptr || count != -1) return 3;
  psgd_tape_free(tape);
  psgd_tape_free(psgd_tape_begin());   // dropped before its end: nothing is written into it any more
  if (psgd_tape_now != nullptr) return 4;
  return 0;
}
"""


def test_a_record_without_memory_is_no_exception(tmp_path):
    """The library is called through C entries, which no exception may leave: the record says that it is not complete."""
    import subprocess

    from powersgd_b200.csrc import build

    try:
        nvcc = build._nvcc()
    except RuntimeError:
        pytest.skip("no CUDA compiler")
    sources, program = [tmp_path / "tape.cu", tmp_path / "memory.cpp"], str(tmp_path / "tape")
    for path, text in zip(sources, (HARNESS, MEMORY)):
        path.write_text(text)
    subprocess.run([nvcc, *build.ARCH, "-std=c++17", "-I", build.HERE, *map(str, sources), "-o", program], check=True)
    assert subprocess.run([program]).returncode == 0


def test_an_interrupt_ends_the_record():
    """Wherever it comes, later launches of the thread are not written down."""
    class Lib:
        open = False

        def psgd_tape_begin(self):
            self.open = True
            raise KeyboardInterrupt   # as the interpreter raises it behind the call

        def psgd_tape_end(self):
            self.open = False
            return -1

        def psgd_tape_free(self, tape):
            pass

    lib = Lib()
    with pytest.raises(KeyboardInterrupt):
        cuda_path._Tape(lib, lambda: None)
    assert not lib.open
