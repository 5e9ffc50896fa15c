"""Which launches may start before their predecessor has ended (host code only, no GPU)."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from powersgd_b200.cuda_path import NativeCompressor


def _orth_flags(comm, early, gather):
    nat = object.__new__(NativeCompressor)
    buf = torch.zeros(4)
    nat.units, nat.chunks, nat.n_units, nat.n_chunks = {"p": buf}, {"p": buf}, {"p": 1}, {"p": 1}
    nat.tiles, nat._orth_part, nat._orth_rinv, nat.comm = SimpleNamespace(max_r=2), buf, buf, comm
    calls = []
    nat._call = lambda name, *args: calls.append((name, args))
    nat._orth("p", buf, buf, [], [], buf if gather else None, early=early)
    (name, args), = calls
    assert name == "psgd_orth_launch"
    return args[-1]


def test_orthonormalisation_overlaps_on_one_worker():
    assert _orth_flags(None, early=False, gather=False) == 2
    assert _orth_flags(None, early=True, gather=False) == 3


@pytest.mark.parametrize("gather", [False, True])
def test_orthonormalisation_keeps_the_plain_order_with_several_workers(gather):
    """A first launch that waits for peers must not have the second one's CTAs resident beside it."""
    assert _orth_flags(SimpleNamespace(ptr=ctypes.c_void_p(8)), early=False, gather=gather) == 0


def test_a_wait_that_ran_out_is_not_put_down_to_the_tensor_cores():
    """The one-pass kernel, which does not use them, reports through the same word."""
    from powersgd_b200.parallel.symm import PowerSGDCommTimeout, StatusWord

    class Word(StatusWord):   # without memory that a GPU can see
        value = 3

        def __init__(self):
            self._host = None

    nat = object.__new__(NativeCompressor)
    nat.comm, nat._status = None, Word()
    with pytest.raises(PowerSGDCommTimeout, match="one-pass kernel") as caught:
        nat.check()
    assert "tensor-core" not in str(caught.value)
    Word.value = 0
    nat.check()


def test_launches_that_may_start_early_promise_nothing_about_what_they_wait_for():
    """A `const __restrict__` parameter may be read through the cache for data that nobody writes while the kernel runs, which does
    not hold for what the launch before it writes. Tables that no launch writes may be declared so."""
    import os
    import re

    import powersgd_b200

    folder = os.path.join(os.path.dirname(powersgd_b200.__file__), "csrc")
    tables, waiting = {"items", "block_item", "block_part", "item_parts"}, 0
    for name in sorted(f for f in os.listdir(folder) if f.endswith(".cu")):
        with open(os.path.join(folder, name)) as fp:
            text = fp.read()
        kernels = list(re.finditer(r"__global__[^;{]*?(\w+_kernel)\(([^{;]*)\)\s*\{", text))
        for kernel, after in zip(kernels, kernels[1:] + [None]):
            body = text[kernel.end() : after.start() if after else len(text)].split("\n}\n")[0]
            if "psgd_wait_for_predecessor" not in body:
                continue
            waiting += 1
            promised = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", kernel.group(2)))
            assert promised <= tables, (name, kernel.group(1), promised - tables)
    assert waiting >= 10, waiting
