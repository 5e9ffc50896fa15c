"""What the native path does while a CUDA graph is being recorded on the current stream.

A recorded launch holds raw addresses: descriptor tables, scratch, factors. Two things follow. What never
changes is put in place at once, beside the recording, and not by a node that every replay would pay for
(`outside_capture`, `to_device`). And everything whose address is recorded is kept for the graph, whatever
its owner binds later (`keep_with_graph`).
"""
from __future__ import annotations

import contextlib
import ctypes
import itertools
from typing import Dict, Optional

import numpy as np
import torch

from . import native


def is_recorded(stream: ctypes.c_void_p) -> bool:
    """Is the current stream, whose handle is `stream`, being recorded? The default stream (handle 0) cannot be,
    so eager loops on it are spared the question, which takes the driver some 2 us while launches are under way."""
    return bool(stream) and torch.cuda.is_current_stream_capturing()


_upload_streams: Dict[torch.device, torch.cuda.Stream] = {}


@contextlib.contextmanager
def outside_capture(device: torch.device):
    """Runs its body at once, whether or not a CUDA graph is being recorded on the current stream: what
    never changes (descriptor tables, cleared counters) is put in place once instead of by a node that
    every replay of the graph pays for (eight copies of 1.3 us each in the step of a small perceptron).
    Under capture the body gets a stream that is not part of it, so that its tensors come from the
    ordinary pool - memory of the graph's own pool may be written by an earlier node of the same graph -
    and is waited for; the thread is in the relaxed capture mode meanwhile, whatever mode the recording
    was begun with (an allocation in the strict one ends it with an error)."""
    if not torch.cuda.is_current_stream_capturing():
        yield
        return
    device = torch.device("cuda", torch.cuda.current_device()) if device.index is None else device
    with native.relaxed_capture():
        while True:
            stream = _upload_streams.setdefault(device, torch.cuda.Stream(device=device))
            with torch.cuda.stream(stream):
                if torch.cuda.is_current_stream_capturing():   # streams are handed out in turn: this one was forked into the capture
                    del _upload_streams[device]
                    continue
                yield
                stream.synchronize()
                return


def to_device(array: np.ndarray, device: torch.device) -> torch.Tensor:
    """Upload a descriptor table: staged through pinned memory with an async copy on the current stream
    (at once and outside the graph while one is being recorded)."""
    release_finished()
    raw = np.ascontiguousarray(array).view(np.uint8).reshape(-1)
    with outside_capture(device):
        pinned = torch.empty(max(raw.size, 1), dtype=torch.uint8).pin_memory()
        pinned.numpy()[: raw.size] = raw
        out = torch.empty(max(raw.size, 1), dtype=torch.uint8, device=device)
        out.copy_(pinned, non_blocking=True)
        out._psgd_pinned_src = pinned
    return out


_kept: Dict[int, tuple] = {}   # by number: what a recorded graph refers to, until the graph is gone
_numbers = itertools.count(1)
_scope: Optional[list] = None


def keep_with_graph(holder: Optional[dict], *objects) -> None:
    """While a CUDA graph is being recorded: `objects` (tensors, or whatever owns memory) stay alive for it.
    Inside a `capture_scope` the program has them. Otherwise `holder` has them, a dict of the object whose
    launches are being recorded (an aggregator must outlive the graphs recorded from it, as the parameters
    must): what that object binds or drops later then takes nothing from under a replay. Without a holder
    the graph itself says when it is gone (a user object whose destructor notes a number); a replay of
    such a graph costs 2 us more."""
    if _scope is not None:
        _scope.append(objects)
    elif holder is not None:
        holder.update((id(o), o) for o in objects)
    else:
        number = next(_numbers)
        _kept[number] = objects
        native.check(
            native.lib().psgd_graph_retain(ctypes.c_longlong(number), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)),
            "psgd_graph_retain",
        )


def release_finished() -> None:
    """Lets go of what only graphs destroyed since the last call referred to. Not while a graph is being
    recorded: giving back pinned memory would end the recording."""
    if not _kept or torch.cuda.is_current_stream_capturing():
        return
    numbers = (ctypes.c_longlong * 256)()
    while True:
        count = native.lib().psgd_graph_released(numbers, len(numbers))
        for number in numbers[:count]:
            _kept.pop(number, None)
        if count < len(numbers):
            return


class capture_scope:
    """`with capture_scope() as keep:` around a CUDA-graph capture collects in `keep` what the graph refers to
    besides the caller's own tensors; store `keep` next to the graph and drop both together. Without it,
    what was recorded lives as long as the aggregator: a program that records again and again on new
    tensors gives back what earlier recordings held by using a scope."""

    def __enter__(self) -> list:
        global _scope
        self._outer = _scope
        _scope = []
        return _scope

    def __exit__(self, *exc):
        global _scope
        _scope = self._outer
