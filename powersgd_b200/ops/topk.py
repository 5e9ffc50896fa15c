"""Magnitude top-k selection with the error-feedback write fused in (csrc/topk.cu).

`topk_abs(x, k, memory=None)` returns `(values, positions)` of the k entries of the flattened
tensor with the largest |x| (order unspecified, positions int32) and, when `memory` is given,
fills it with x where the taken entries are zeroed. On CPU (or on CUDA without the native
library when PSGD_B200_ALLOW_FALLBACK=1 allows it; otherwise that is an error) the same result
comes from `torch.topk` (gradient_reducers.py:240-253 is the reference sequence).
"""
from __future__ import annotations

import ctypes
import threading
from typing import Optional, Tuple

import torch

from . import native, scan
from .recording import is_recorded, keep_with_graph, outside_capture, release_finished

# Scratch (histograms, counters, lists, a barrier word) belongs to one stream, whose order keeps the calls that
# share it apart, and the launches of a call go onto it in one piece: two streams, or two threads on one stream, that
# share counters would hand out places beyond the end of a list. What is dropped here goes back to the
# allocator of the same stream, behind the launches that use it.
_launching = threading.RLock()
MOST_STREAMS = 64
_workspaces: dict = {}


def _current_stream() -> ctypes.c_void_p:
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()))


def _of_stream(pool: dict, device: torch.device, stream: ctypes.c_void_p, make) -> torch.Tensor:
    key = (device, stream.value)
    if key not in pool:
        if len(pool) >= MOST_STREAMS:
            del pool[next(iter(pool))]
        pool[key] = make()
    return pool[key]


def topk_abs(x: torch.Tensor, k: int, memory: Optional[torch.Tensor] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    flat = x.reshape(-1)
    n = flat.numel()
    k = int(k)
    if flat.is_cuda and native.use_for_cuda() and flat.dtype == torch.float32 and flat.is_contiguous() and (
        memory is None or (memory.is_contiguous() and memory.dtype == torch.float32)
    ):
        lib = native.lib()
        stream = _current_stream()
        make = lambda: torch.zeros(lib.psgd_topk_workspace_ints(), dtype=torch.int32, device=flat.device)  # noqa: E731
        values = torch.empty(k, dtype=torch.float32, device=flat.device)
        positions = torch.empty(k, dtype=torch.int32, device=flat.device)
        with _launching:
            if is_recorded(stream):   # a graph gets counters of its own, see topk_abs_many
                ws = make()
                keep_with_graph(None, ws)
            else:
                ws = _of_stream(_workspaces, flat.device, stream, make)
            code = lib.psgd_topk_abs(
                ctypes.c_void_p(flat.data_ptr()), ctypes.c_longlong(n), ctypes.c_longlong(k), ctypes.c_void_p(ws.data_ptr()),
                ctypes.c_void_p(values.data_ptr()), ctypes.c_void_p(positions.data_ptr()),
                ctypes.c_void_p(0 if memory is None else memory.data_ptr()), stream,
            )
        native.check(code, "psgd_topk_abs")
        return values, positions
    _, idx = torch.topk(flat.abs(), k, sorted=False)
    values = flat[idx].contiguous()
    if memory is not None:
        memory.copy_(x)
        memory.view(-1)[idx] = 0.0
    return values, idx.to(torch.int32)


_many_cache: dict = {}
MOST_LISTS = 8   # of tensors, each on one stream, whose tables are kept
BLOCKS = 3 * 148
CANDIDATES = 2048   # room for candidates per tensor, besides what the length of the list allows (0: none)


def topk_abs_many(tensors, ks, memories=None, outs=None) -> Tuple[torch.Tensor, torch.Tensor]:
    """`topk_abs` for a list of tensors in four launches (csrc/topk.cu, psgd_topk_abs_many).

    Returns flat `(values, positions)`: tensor i's `ks[i]` pairs start at `sum(ks[:i])`; positions
    are int32 indices into the flattened tensor i. `memories[i]`, when given, receives tensor i with
    the taken entries zeroed. `outs[i]`, when given, receives the taken entries of tensor i at their places and
    zeros elsewhere: what `sparse_combine` makes of one worker's pairs, without a pass of its own where `outs` lie apart
    from what is read. Falls back to one `topk_abs` per tensor off the GPU."""
    ks = [int(k) for k in ks]
    total = sum(ks)
    tensors = list(tensors)
    mems = list(memories) if memories is not None else [None] * len(tensors)
    device = tensors[0].device
    # contiguous: their memory is then the flattened tensor
    native_ok = device.type == "cuda" and native.use_for_cuda() and scan.usable(tensors, True) and scan.usable([m for m in mems if m is not None], True)
    if not native_ok:
        values = torch.empty(total, dtype=torch.float32, device=device)
        positions = torch.empty(total, dtype=torch.int32, device=device)
        at = 0
        for t, k, m in zip(tensors, ks, mems):
            v, p = topk_abs(t, k, memory=m)
            values[at : at + k], positions[at : at + k] = v, p
            at += k
        if outs is not None:
            _combine_own(values, positions, ks, list(outs))
        return values, positions
    values = torch.empty(total, dtype=torch.float32, device=device)
    positions = torch.empty(total, dtype=torch.int32, device=device)
    outs = None if outs is None else list(outs)
    dense = outs is not None and scan.usable(outs, True)
    with _launching:
        dense = _select(tensors, ks, mems, outs if dense else None, values, positions) and dense
    if outs is not None and not dense:
        _combine_own(values, positions, ks, outs)
    return values, positions


def _combine_own(values: torch.Tensor, positions: torch.Tensor, ks, outs) -> None:
    ends, at = [], 0
    for k in ks:
        at += k
        ends.append(at)
    sparse_combine(values.view(1, -1), positions.view(1, -1), outs, ends, 1.0)


def _apart(outs, sizes, read) -> bool:
    """Do the tensors `outs` have the numbers of elements `sizes`, and no byte in common with each other or with the tensors `read`?
    A launch may write one tensor's part of `outs` while another's is still to be read."""
    import numpy as np

    if any(o.numel() != n for o, n in zip(outs, sizes)):
        return False
    start = np.array([o.data_ptr() for o in outs], dtype=np.uint64)
    order = np.argsort(start, kind="stable")
    start, end = start[order], (start + 4 * np.array(sizes, dtype=np.uint64))[order]
    if (end[:-1] > start[1:]).any():
        return False
    first = np.array([t.data_ptr() for t in read], dtype=np.uint64)
    last = first + 4 * np.array([t.numel() for t in read], dtype=np.uint64)
    before = np.searchsorted(start, last, side="left")   # how many begin before the end of what is read; the last of them ends last
    return not ((before > 0) & (end[np.maximum(before, 1) - 1] > first)).any()


def _select(tensors, ks, mems, outs, values: torch.Tensor, positions: torch.Tensor) -> bool:
    """The launches; are `outs` written as well?"""
    import numpy as np

    lib = native.lib()
    device = tensors[0].device
    stream = _current_stream()
    key = (device, stream.value, scan.addresses(tensors), scan.addresses(mems), scan.sizes(tensors), tuple(ks), scan.addresses(outs),
           None if outs is None else scan.sizes(outs))   # (an output of another length is not written by these launches)
    # a recorded call gets tables and counters of its own: the cache may drop an entry at any time, and a
    # replay may run beside an eager call on the same tensors
    recorded = is_recorded(stream)
    entry = None if recorded else _many_cache.get(key)
    # (open: a call was broken off, and the half of the workspace that the next one counts in may not be cleared)
    if entry is None or entry["open"]:
        release_finished()
        dtype = np.dtype([("x", np.uint64), ("memory", np.uint64), ("n", np.int64), ("k", np.int64), ("out_off", np.int64),
                          ("cand_off", np.int64), ("cap", np.int64), ("out", np.uint64)])
        if dtype.itemsize != int(lib.psgd_topk_item_bytes()):
            raise RuntimeError("top-k item record out of sync with the native library")
        items = np.zeros(len(tensors), dtype=dtype)
        block_item, block_part, parts = [], [], []
        at, room, total_n = 0, 0, max(1, sum(t.numel() for t in tensors))
        dense = outs is not None and _apart(outs, [t.numel() for t in tensors], tensors + [m for m in mems if m is not None])
        for i, (t, k, m) in enumerate(zip(tensors, ks, mems)):
            n = t.numel()
            if not (0 < k <= n < (1 << 31)):
                raise ValueError(f"topk_abs_many: need 0 < k <= n < 2^31 (k = {k}, n = {n})")
            # candidates: entries that agree with the threshold in their leading 11 bits (an eighth of an octave), some
            # 0.75 k in a normal distribution's tail. One block walks a tensor's list, 1.2 us per 1000 entries; a tensor with
            # more of them than that goes the long way, some 1.2 us per million entries of the whole list of tensors.
            # Room for half of what would break even. us per replayed call, long way / lists: 1 M, 1 700 candidates 25 / 25,
            # 12 600 26 / 38; 4 M, 3 800 43 / 38, 27 000 45 / 63; 16 M, 15 000 75 / 77, 820 000 (uniform) 76 / 849; 50 M, 47 000
            # 203 / 197, 81 000 203 / 238; 62 tensors of 11 M, 3 900 in the largest 68 / 54, 33 000 73 / 91
            cap = min(n, CANDIDATES + total_n // 2048) if CANDIDATES else 0
            items[i] = (t.data_ptr(), 0 if m is None else m.data_ptr(), n, k, at, room, cap, outs[i].data_ptr() if dense else 0)
            at, room = at + k, room + cap
            # blocks of 512 threads with at least 16 elements each, three per SM for the whole list, as many as run at a time: every
            # block pays for its histogram (zeroing, choosing the digits so far, adding it up), and a few blocks more are a
            # round of their own. us per pass with 370 / 444 / 592 / 888 blocks: ResNet-18 52.7 / 51.5 / 54.7 / 56.2, 16 M + 0.7 M entries
            # 72.9 / 70.9 / 74.9 / 77.3, 48 M 234 / 217 / 217 / 219
            nparts = max(1, min(-(-n // (512 * 16)), BLOCKS * n // total_n))
            parts.append(nparts)
            block_item += [i] * nparts
            block_part += list(range(nparts))
        to_dev = lambda a: torch.from_numpy(a.view(np.uint8) if a.dtype.names else a).to(device)  # noqa: E731
        with outside_capture(device):
            entry = {
                "items": to_dev(items), "block_item": to_dev(np.asarray(block_item, dtype=np.int32)),
                "block_part": to_dev(np.asarray(block_part, dtype=np.int32)), "parts": to_dev(np.asarray(parts, dtype=np.int32)),
                "nblocks": len(block_item), "dense": dense, "turn": 0, "open": False,
                "cand_v": torch.empty(max(room, 1), dtype=torch.float32, device=device), "cand_p": torch.empty(max(room, 1), dtype=torch.int32, device=device),
                # one half per call in turn: a call clears the other for the next. (A recorded call clears its own.)
                "ws": torch.zeros(2 * len(tensors) * int(lib.psgd_topk_workspace_ints()), dtype=torch.int32, device=device),
            }
        if recorded:
            keep_with_graph(None, entry)
        else:
            # the tables hold addresses and lengths only, and the key is exactly those: an entry stays
            # valid for whatever tensors present the same addresses again, so no tensor is kept alive
            if len(_many_cache) >= MOST_LISTS:
                _many_cache.clear()
            _many_cache[key] = entry
    vp = ctypes.c_void_p
    half = 2 * entry["ws"].numel()   # in bytes
    turn, base = entry["turn"], entry["ws"].data_ptr()
    entry["open"] = True
    code = lib.psgd_topk_abs_many(
        vp(entry["items"].data_ptr()), len(tensors), vp(entry["block_item"].data_ptr()), vp(entry["block_part"].data_ptr()),
        vp(entry["parts"].data_ptr()), entry["nblocks"], vp(base + turn * half), vp(0 if recorded else base + (1 - turn) * half),
        vp(entry["cand_v"].data_ptr()), vp(entry["cand_p"].data_ptr()), vp(values.data_ptr()), vp(positions.data_ptr()), stream,
    )
    native.check(code, "psgd_topk_abs_many")
    entry["turn"], entry["open"] = 1 - turn, False
    return entry["dense"]


_SEG_DTYPE = None
_combine_scratch = {}
_segment_cache: dict = {}


def sparse_combine(all_values: torch.Tensor, all_positions: torch.Tensor, outs, ends, divisor: float) -> None:
    """outs[s] <- sum over workers of value / divisor of the (value, position) pairs of segment s, scattered.

    `all_values` / `all_positions`: [workers, K] float32 / int32 (rows as all-gathered); segment s
    owns columns [ends[s-1], ends[s]) of every row, its positions index into the flattened
    `outs[s]`. Positions are unique within a row's segment. On CUDA one cooperative launch zeroes
    the outputs and applies the workers in rank order (csrc/topk.cu), so replicas stay
    bit-identical; elsewhere the same sum runs as one `index_add_` per worker
    (gradient_reducers.py:262-271)."""
    workers = all_values.shape[0]
    use_native = (
        all_values.is_cuda and native.use_for_cuda() and all_values.dtype == torch.float32 and all_positions.dtype == torch.int32
        and all_values.is_contiguous() and all_positions.is_contiguous()
        and scan.usable(outs, True)
    )
    if use_native:
        with _launching:
            _combine(all_values, all_positions, outs, ends, divisor)
        return
    start = 0
    for out, end in zip(outs, ends):
        out.zero_()
        flat = out.view(-1)
        for w in range(workers):
            flat.index_add_(0, all_positions[w, start:end].long(), all_values[w, start:end] / divisor)
        start = end


def _combine(all_values: torch.Tensor, all_positions: torch.Tensor, outs, ends, divisor: float) -> None:
    global _SEG_DTYPE
    import numpy as np

    workers, per_worker = all_values.shape
    lib = native.lib()
    cap = int(lib.psgd_sparse_combine_max_segments())
    if _SEG_DTYPE is None:
        _SEG_DTYPE = np.dtype([("out", np.uint64), ("numel", np.int64), ("end", np.int64)])
    device = all_values.device
    stream = _current_stream()

    def words() -> torch.Tensor:   # [grid barrier, status]
        with outside_capture(device):
            return torch.zeros(2, dtype=torch.int32, device=device)

    scratch = _of_stream(_combine_scratch, device, stream, words)
    barrier = scratch
    # tables of addresses and lengths, kept by exactly those (as the selection's above, recorded calls
    # included): building and uploading one stalls the host until the selection has run
    key = (device, scan.addresses(outs), scan.sizes(outs), tuple(ends))
    recorded = is_recorded(stream)
    tables = None if recorded else _segment_cache.get(key)
    if tables is None:
        release_finished()
        tables = []
        with outside_capture(device):
            for first in range(0, len(outs), cap):
                chunk = list(range(first, min(first + cap, len(outs))))
                segs = np.zeros(len(chunk), dtype=_SEG_DTYPE)
                base = ends[first - 1] if first else 0
                for j, s in enumerate(chunk):
                    segs[j] = (outs[s].data_ptr(), outs[s].numel(), ends[s] - base)
                tables.append((torch.from_numpy(segs.view(np.uint8)).to(device, non_blocking=False), len(chunk), base, ends[chunk[-1]] - base))
            if recorded:
                barrier = torch.zeros(1, dtype=torch.int32, device=device)
        if recorded:
            keep_with_graph(None, tables, barrier, scratch)
        else:
            if len(_segment_cache) >= 4:
                _segment_cache.clear()
            _segment_cache[key] = tables
    for segs_dev, count, base, width in tables:
        vals = all_values if (base == 0 and width == per_worker) else all_values[:, base : base + width].contiguous()
        poss = all_positions if (base == 0 and width == per_worker) else all_positions[:, base : base + width].contiguous()
        code = lib.psgd_sparse_combine_launch(
            ctypes.c_void_p(vals.data_ptr()), ctypes.c_void_p(poss.data_ptr()), int(workers), ctypes.c_longlong(width),
            ctypes.c_void_p(segs_dev.data_ptr()), count, ctypes.c_float(divisor),
            ctypes.c_void_p(barrier.data_ptr()), ctypes.c_void_p(scratch.data_ptr() + 4), stream,
        )
        native.check(code, "psgd_sparse_combine_launch")
        if not recorded:
            segs_dev.record_stream(torch.cuda.current_stream())


def sparse_combine_status(device) -> int:
    """0 unless a grid barrier of `sparse_combine` gave up on `device` (reads the device words: synchronises)."""
    return max((int(words[1].item()) for (of, _stream), words in list(_combine_scratch.items()) if of == torch.device(device)), default=0)
