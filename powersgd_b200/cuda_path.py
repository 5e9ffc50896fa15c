"""Drives the native sm_100a kernels for the compressor core and the flat all-reduce.

Per optimizer step the reference issues several hundred small PyTorch ops
(powersgd/powersgd.py:146-235). Here a step is, for T half-iterations:

    T x [ orthonormalise (2 launches; multi-GPU: the first one also gathers the factor the previous
          product pushed, i.e. it is the consumer of the in-kernel all-reduce)
          -> grouped product (1 launch; multi-GPU: its epilogue pushes the fresh factor to every peer) ]
      ->  decompress + error feedback (+ SGD) (1 launch; multi-GPU: gathers the last factor itself)

over ALL shape groups at once. The gradient matrices are addressed in place through a
pointer table (no `torch.stack`, no un-batching copies), the deflation between half-iterations
is algebraic (small r x r corrections), and the residual is written exactly once.

Factor bookkeeping for half-iteration t of a step (left = the P side is the input):

    left :  Lloc = Lsum = orth(P)      Rloc = local M^T P      Rsum = sum over workers
    right:  Rloc = Rsum = orth(Q)      Lloc = local M Q        Lsum = sum over workers

    residual = M - sum_t Lloc_t Rloc_t^T        update = (1/W) sum_t Lsum_t Rsum_t^T
"""
from __future__ import annotations

import contextlib
import ctypes
import heapq
import os
import weakref
from typing import Dict, List, Optional, Sequence, Tuple

import numpy as np
import torch
import torch.distributed as dist

from .ops import layout, native, scan
from .ops.recording import capture_scope, is_recorded, keep_with_graph, outside_capture  # noqa: F401  (capture_scope: for callers)
from .ops.recording import to_device as _to_device
from .utils import is_dense, like_strided, same_layout, world_size


class _Range:
    """A named phase of `aggregate()`: an NVTX range when PSGD_B200_NVTX=1 (phase names show up
    in profiler timelines), a CUDA-event pair appended to `_Range.events` when a benchmark set
    that list (per-phase device times), free otherwise."""

    enabled = os.environ.get("PSGD_B200_NVTX", "0") == "1"
    events: Optional[list] = None

    def __init__(self, name: str):
        self.name = name

    def __enter__(self):
        if self.enabled:
            torch.cuda.nvtx.range_push(self.name)
        if _Range.events is not None:
            self._start = torch.cuda.Event(enable_timing=True)
            self._start.record()

    def __exit__(self, *exc):
        if _Range.events is not None:
            stop = torch.cuda.Event(enable_timing=True)
            stop.record()
            _Range.events.append((self.name, self._start, stop))
        if self.enabled:
            torch.cuda.nvtx.range_pop()


def _stream_ptr() -> ctypes.c_void_p:
    return ctypes.c_void_p(torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice()))


def _ptr(t: Optional[torch.Tensor]) -> ctypes.c_void_p:
    return ctypes.c_void_p(0 if t is None else t.data_ptr())


def _ptr_array(tensors: Sequence[torch.Tensor]):
    arr = (ctypes.c_void_p * max(len(tensors), 1))()
    for i, t in enumerate(tensors):
        arr[i] = t.data_ptr()
    return arr


def _split_even(total: int, max_chunk: int, multiple: int) -> List[Tuple[int, int]]:
    """Cut [0, total) into near-equal chunks of at most `max_chunk`, starts on `multiple`."""
    return _split_parts(total, -(-total // max_chunk), multiple)


def _split_parts(total: int, parts: int, multiple: int) -> List[Tuple[int, int]]:
    """Cut [0, total) into at most `parts` near-equal chunks, starts on `multiple`."""
    if parts <= 1:
        return [(0, total)]
    size = -(-total // parts)
    size = -(-size // multiple) * multiple
    out, start = [], 0
    while start < total:
        out.append((start, min(size, total - start)))
        start += size
    return out


def _split_count(total: int, max_chunk: int, multiple: int) -> int:
    """len(_split_even(total, max_chunk, multiple))"""
    if total <= max_chunk:
        return 1
    size = -(-total // -(-total // max_chunk))
    return -(-total // (-(-size // multiple) * multiple))


class TilePlan:
    """Static tile lists (independent of tensor addresses) for one CompressionPlan."""

    def __init__(self, plan, lib):
        self.plan, self._lib = plan, lib
        mats = []  # (group index, position, compressed-list index)
        for gi, g in enumerate(plan.groups):
            for pos, idx in enumerate(g.members):
                mats.append((gi, pos, idx))
        self.mats = mats
        self.max_r = max((g.r for g in plan.groups), default=1)
        if self.max_r > layout.MAX_RANK:
            raise ValueError(f"rank {self.max_r} exceeds the compiled maximum {layout.MAX_RANK}")
        self.rt = lib.psgd_gemm_template_rank(self.max_r)
        self.total_elems = sum(g.n * g.m * g.batch for g in plan.groups)
        self._nt_rows_cap = lib.psgd_gemm_nt_max_rows(self.max_r)
        self.nt_rows, self.nt_tall_rows = min(self._nt_rows_cap, 128), 256   # chosen anew by every `build`
        self.nn_rows = lib.psgd_gemm_nn_tile_rows(self.max_r)
        self.nn_cols_cap = lib.psgd_gemm_nn_max_cols(self.max_r)
        self.rp_tc = lib.psgd_gemm_tc_rank_pad(self.max_r)
        self.fin_tc_ok = False  # set by the compressor: (half-iterations x rank) fits the tensor-core finalize
        self.fin_rows = 32      # set by the compressor: height of a finalize strip (multiple of 32)

    def build(self, vec_widths: Sequence[int], tc_flags: Optional[Sequence[bool]] = None):
        """Tile arrays for the CUDA-core kernels (key "f"; every tile carries the access width of
        its matrix: 4, 2 or 1 floats) and, for the matrices flagged in `tc_flags`, tensor-core
        tiles (key "tc")."""
        nt = {"f": [], "tc": []}
        nn = {"f": [], "tc": []}
        fin = {"f": [], "tc": []}
        ticket = 0
        nt_slots = nn_slots = tc_slots = 0
        tc_flags = tc_flags or [False] * len(self.mats)
        # K extent of one tensor-core tile: long enough to amortise the pipeline ramp and the
        # epilogue, short enough that a small model still fills the GPU, and such that the last
        # wave of CTAs is nearly full (the block scheduler runs TC_CTAS_PER_SM per SM at a time)
        tc_mats = [self.plan.groups[gi] for (gi, _p, _i), f in zip(self.mats, tc_flags) if f]
        tc_k_nt, tail_nt = self._tc_extents(tc_mats, transposed=True)
        tc_k_nn, tail_nn = self._tc_extents(tc_mats, transposed=False)
        tc_nt = tc_nn = 0   # output blocks so far
        self._pick_nt_rows([self.plan.groups[gi] for (gi, _p, _i), f in zip(self.mats, tc_flags) if not f])
        for mi, (gi, _pos, _idx) in enumerate(self.mats):
            g = self.plan.groups[gi]
            v = int(vec_widths[mi])
            if tc_flags[mi] and self.fin_tc_ok:
                fin["tc"].append((mi, g.n, 128, g.m, 64, v))
            else:
                fin["f"].append((mi, g.n, self.fin_rows, g.m, 128, v))
            if tc_flags[mi]:
                row_blocks, col_blocks = _split_even(g.n, tc_k_nt, 32), _split_even(g.m, tc_k_nn, 32)
                whole_rows, whole_cols = row_blocks, col_blocks
                for c0 in range(0, g.m, 128):
                    if tail_nt:
                        row_blocks = _split_parts(g.n, tail_nt[tc_nt], 32) if tc_nt in tail_nt else whole_rows
                        tc_nt += 1
                    for si, (r0, rows) in enumerate(row_blocks):
                        nt["tc"].append((mi, r0, rows, c0, min(128, g.m - c0), si, len(row_blocks), ticket, tc_slots, v, (0, 0)))
                    ticket += 1
                    tc_slots += len(row_blocks)
                for r0 in range(0, g.n, 128):
                    if tail_nn:
                        col_blocks = _split_parts(g.m, tail_nn[tc_nn], 32) if tc_nn in tail_nn else whole_cols
                        tc_nn += 1
                    for si, (c0, cols) in enumerate(col_blocks):
                        nn["tc"].append((mi, r0, min(128, g.n - r0), c0, cols, si, len(col_blocks), ticket, tc_slots, v, (0, 0)))
                    ticket += 1
                    tc_slots += len(col_blocks)
                continue
            row_blocks = _split_even(g.n, self._nt_tile_rows(g.n), 1)
            for c0 in range(0, g.m, 128):
                cols = min(128, g.m - c0)
                for si, (r0, rows) in enumerate(row_blocks):
                    nt["f"].append((mi, r0, rows, c0, cols, si, len(row_blocks), ticket, nt_slots, v, (0, 0)))
                ticket += 1
                nt_slots += len(row_blocks)
            col_blocks = _split_even(g.m, self.nn_cols_cap, 128)
            for r0 in range(0, g.n, self.nn_rows):
                rows = min(self.nn_rows, g.n - r0)
                for si, (c0, cols) in enumerate(col_blocks):
                    nn["f"].append((mi, r0, rows, c0, cols, si, len(col_blocks), ticket, nn_slots, v, (0, 0)))
                ticket += 1
                nn_slots += len(col_blocks)
        self.n_tickets = max(ticket, 1)
        self.partial_floats = max(nt_slots * 128 * self.rt, nn_slots * self.nn_rows * self.rt, 1)
        self.partial_tc_floats = max(tc_slots * 128 * self.rp_tc, 1)

        def arr(items):
            return np.array(items, dtype=layout.TILE_DTYPE) if items else np.zeros(0, dtype=layout.TILE_DTYPE)

        return {
            "nt": {k: arr(v) for k, v in nt.items()},
            "nn": {k: arr(v) for k, v in nn.items()},
            # last rows first: some of what the product before has read last is still in the L2 cache. us per pass, first rows first / last
            # rows first: LSTM step 212.7 / 210.9, ResNet-18's recorded step 103.2 / 102.6, 50257 x 1024 at rank 16 427.7 / 426.2
            "fin": {k: self._grids(v)[::-1].copy() if v else arr(v) for k, v in fin.items()},
        }

    @staticmethod
    def _grids(matrices: Sequence[Tuple[int, int, int, int, int, int]]) -> np.ndarray:
        """Tiles of `rows` x `cols` over every (index, n, rows, m, cols, access width) of a list, row by row. By array
        operations over all matrices at once; one by one up to some 40 tiles, which the array operations cost alone."""
        if sum(-(-n // rows) * -(-m // cols) for _mi, n, rows, m, cols, _v in matrices) <= 40:
            return np.array([(mi, r0, min(rows, n - r0), c0, min(cols, m - c0), 0, 1, 0, 0, v, (0, 0))
                             for mi, n, rows, m, cols, v in matrices for r0 in range(0, n, rows) for c0 in range(0, m, cols)], dtype=layout.TILE_DTYPE)
        mat, n, rows, m, cols, vec = np.array(matrices, dtype=np.int32).reshape(-1, 6).T
        across = -(-m // cols)
        count = -(-n // rows) * across
        of = np.repeat(np.arange(len(count)), count)
        at = np.arange(len(of), dtype=np.int32) - (np.cumsum(count) - count)[of]
        down, right = np.divmod(at, across[of])
        row0, col0 = down * rows[of], right * cols[of]
        tiles = np.zeros((len(of), layout.TILE_DTYPE.itemsize // 4), dtype=np.int32)
        for name, values in (("mat", mat[of]), ("row0", row0), ("rows", np.minimum(rows[of], n[of] - row0)), ("col0", col0),
                             ("cols", np.minimum(cols[of], m[of] - col0)), ("nsplit", 1), ("vec", vec[of])):
            tiles[:, layout.TILE_DTYPE.fields[name][1] // 4] = values
        return tiles.view(layout.TILE_DTYPE).reshape(-1)

    def _nt_tile_rows(self, n: int) -> int:
        # tall matrices: never more than 160 partial tiles per column block (the kernel walks a tile that is
        # taller than its staging buffer in chunks)
        return max(self.nt_rows if n <= 4096 else self.nt_tall_rows, -(-(-(-n // 160)) // 128) * 128)

    def _pick_nt_rows(self, groups) -> None:
        """Rows of an NT tile (`groups`: the matrices of the CUDA-core launch, one entry each): 128 or 256, and
        256 or 512 above 4096 rows. Twice as many halve what a tile costs besides its loads (start, staging,
        the sum over the warps, the hand-over), as long as the launch still fills some half of the places that
        the SMs have for its CTAs (three per SM up to template rank 4, two above); only its own tiles count,
        not the elements of the model, most of which may go to the tensor cores. Of the tall matrices only
        their own tiles count: among many short ones a few tall tiles end last. Measured (us per launch, data in
        L2, tiles at the larger height), 128 / 256 rows: 186 (3 x 1001x777 + 2 x 515x2049, rank 3) 9.4 / 11.1, 192
        (6 x 1024x1001, rank 2) 8.1 / 9.8, 256 (8 of them) 11.9 / 9.8, 378 (ResNet-18) 12.8 / 10.9; rank 8, 256: 16.1 /
        13.4; 36 (2 x 700x650 beside two matrices of 33 M elements) 6.0 / 8.1. 256 / 512 rows: 204 (17000x650, rank
        4) 17.7 / 18.8, 252 (21001x650) 26.3 / 19.5, 786 (the LSTM model) 46.2 / 43.1; 323 of which 44 tall 12.4 /
        16.8. Over 200 random lists of matrices the choice is on average 2 % slower than the best of the four
        (5 % when the elements of the model decided), at worst 27 %."""
        enough, enough_tall = (250, 220) if self.rt <= 4 else (150, 80)

        def tiles(rows: int, tall_rows: int, above: int = 0) -> int:
            self.nt_rows, self.nt_tall_rows = min(self._nt_rows_cap, rows), tall_rows
            return sum(-(-g.m // 128) * -(-g.n // self._nt_tile_rows(g.n)) for g in groups if g.n > above)

        rows = 256 if tiles(256, 256) >= enough else 128
        if tiles(rows, 512, above=4096) < enough_tall:
            tiles(rows, 256)

    TC_CTAS_PER_SM = 2
    TC_CHAIN = 512         # rows that a product kernel adds up in the tensor core at a time
    TC_MAX_EXTENT = 8192   # rows of a tile; from some thousand on its overhead does not count any more
    # prologue + epilogue of a tile (~4 us), in units of streamed K rows (~0.03 us each): measured
    # as rounds x (overhead + rows) over tile extents 512 ... 4096 on 4 x 4096^2
    TC_TILE_OVERHEAD_ROWS = 136

    # The same above rank 8 for lists of one to three rounds. Of 330 (from rounds of 352 to 1408 rows alone) to 900, 500 tells best which
    # plans are faster: over 71 products of random lists at rank 11 to 32 that it changes they take 0.87 of the time with the extent of
    # `_pick_tc_k`, at worst 1.03; plans less than a tenth better by it were 9 % slower to 6 % faster.
    TC_ROUND_OVERHEAD_ROWS = 500

    def _tc_extents(self, groups, transposed: bool) -> Tuple[int, Dict[int, int]]:
        """K extent of the tiles, and how many tiles the last output blocks of 128 (by number, in the order of `build`) are cut in if
        not by that. In lists of one to three rounds of resident CTAs what does not fill the last round is cut finer, so that it
        does: 50257 x 1024 at rank 16, P = M Q: 393 blocks in 393 tiles 74 us, in 786 80 (the extent that fills its rounds best), 296 whole
        ones and 97 in three 68. Above, the scheduler evens rounds out by itself (GPT-2 medium, five to eight rounds: 286 -> 277 us for
        one product, 253 -> 269 for the other). A plan is taken for the time at which its last CTA ends, the tiles handed out in
        their order to the first place that is free, and only where that is a tenth earlier than with the extent of `_pick_tc_k`:
        matrices of different lengths have tiles of different lengths, and a few long ones among them keep their places alone. Nor
        may it cost precision (`_tc_error`): 2 x 25718x460 at rank 16, M Q, 3.1e-6 from 64 bits in sums of 460, 1.8e-6 in sums of 232."""
        slots = 148 * self.TC_CTAS_PER_SM
        plain = self._pick_tc_k(groups, transposed)
        blocks = [((g.n if transposed else g.m), -(-(g.m if transposed else g.n) // 128)) for g in groups]   # of (length, number)
        # (above rank 8: at 8 two half-iterations leave directions of nearly equal size, where another order of a sum shows in later steps)
        if (self.rp_tc <= 8 or os.environ.get("PSGD_B200_TC_K")
                or not slots < sum(number * _split_count(length, plain, 32) for length, number in blocks) <= 3 * slots):
            return plain, {}
        lengths, work = {length for length, _number in blocks}, sum(length * number for length, number in blocks)
        error = lambda k: [self._tc_error(length, k) for length in lengths]  # noqa: E731
        longest, usual, best = max(lengths), error(plain), (plain, {})
        end = 0.9 * self._tc_end(self._tc_runs(blocks, plain, {}), float("inf"))
        pieces = -(-longest // self.TC_MAX_EXTENT)
        for k in [plain] + [-(-longest // p) for p in range(pieces, pieces + 8)]:
            tiles = sum(number * _split_count(length, k, 32) for length, number in blocks)
            if work + tiles * self.TC_ROUND_OVERHEAD_ROWS >= end * slots or any(e > before for e, before in zip(error(k), usual)):
                continue
            tail = self._tc_tail(blocks, k, tiles)
            earlier = self._tc_end(self._tc_runs(blocks, k, tail), end)
            if earlier < end:
                best, end = (k, tail), earlier
        return best

    def _tc_error(self, length: int, k: int) -> int:
        """Grows with the error of sums of `length` in tiles of an extent of `k`. The tensor core truncates as it adds, so a chain of n terms,
        the sum of which grows as the root of n, is off by the 3/2th power of n; chains are added up rounded, their errors independent."""
        def of(tile: int) -> int:
            whole, rest = divmod(tile, self.TC_CHAIN)
            return whole * self.TC_CHAIN ** 3 + rest ** 3

        tiles = _split_count(length, k, 32)
        size = length if tiles == 1 else _split_even(length, k, 32)[0][1]
        return (tiles - 1) * of(size) + of(length - (tiles - 1) * size)

    def _tc_tail(self, blocks: Sequence[Tuple[int, int]], k: int, tiles: int) -> Dict[int, int]:
        """The output blocks whose tiles would make up the last round of `tiles` at an extent of `k`, and in how many tiles they fill it."""
        slots = 148 * self.TC_CTAS_PER_SM
        rest = tiles % slots
        finer, at, tail = slots // rest if rest else 1, sum(number for _length, number in blocks), {}
        for length, number in reversed(blocks):
            if finer == 1 or rest <= 0:
                break
            parts = _split_count(length, k, 32)
            number = min(number, -(-rest // parts))
            at, rest = at - number, rest - number * parts
            tail.update(dict.fromkeys(range(at, at + number), _split_count(length, max(128, -(-length // (parts * finer))), 32)))
        return tail

    def _tc_runs(self, blocks: Sequence[Tuple[int, int]], k: int, tail: Dict[int, int]) -> List[Tuple[int, int]]:
        """What the tiles of a plan take, in rows, and how many of them do, in their order (but for the last tiles of the blocks of a
        matrix, which are counted behind the others)."""
        runs, at, overhead = [], 0, self.TC_ROUND_OVERHEAD_ROWS

        def add(length: int, parts: int, number: int) -> None:
            size = -(-length // (32 * parts)) * 32 if parts > 1 else length   # (as `_split_parts`)
            whole, rest = divmod(length, size)
            runs.append((overhead + size, whole * number))
            if rest:
                runs.append((overhead + rest, number))

        first = min(tail, default=sum(number for _length, number in blocks))   # of the blocks that are cut finer, all behind it
        for length, number in blocks:
            usual = min(max(first - at, 0), number)
            if usual:
                add(length, -(-length // k), usual)
            if usual < number:   # (alike within a matrix)
                add(length, tail[at + usual], number - usual)
            at += number
        return runs

    def _tc_end(self, runs: Sequence[Tuple[int, int]], limit: float) -> float:
        """When the last CTA ends, in rows; `limit` if that is not before it."""
        free, ends = {0: 148 * self.TC_CTAS_PER_SM}, [0]   # how many places are free from when on; a heap of these times
        for t, number in runs:
            while number:
                first = ends[0]
                end, taken = first + t, min(number, free[first])
                if end >= limit:
                    return limit
                number -= taken
                free[first] -= taken
                if not free[first]:
                    del free[heapq.heappop(ends)]
                if end in free:
                    free[end] += taken
                else:
                    free[end] = taken
                    heapq.heappush(ends, end)
        return max(ends)

    def _pick_tc_k(self, groups, transposed: bool) -> int:
        if not groups:
            return 512
        if os.environ.get("PSGD_B200_TC_K"):
            return int(os.environ["PSGD_B200_TC_K"])  # tuning knob: fixed K extent (a multiple of 32)
        slots = 148 * self.TC_CTAS_PER_SM
        best, best_score = 512, -1.0
        extents: Dict[int, int] = {}   # output blocks by length of their sums
        for g in groups:
            k_len, out_len = (g.n, g.m) if transposed else (g.m, g.n)
            extents[k_len] = extents.get(k_len, 0) + -(-out_len // 128)
        longest = max(extents)
        ks = np.arange(256, max(256, min(self.TC_MAX_EXTENT, -(-longest // 32) * 32)) + 1, 32)
        tiles = 0
        for k_len, blocks in extents.items():   # (`_split_count` of all of them)
            size = -(-k_len // -(-k_len // ks))
            tiles = tiles + blocks * -(-k_len // (-(-size // 32) * 32))
        waves = -(-tiles // slots)
        scores = tiles / (waves * slots) * ks / (ks + self.TC_TILE_OVERHEAD_ROWS)
        for k, score in zip(ks.tolist(), scores.tolist()):
            if score > best_score + 1e-9:
                best, best_score = k, score
        return best

    # What the one-pass kernel takes for a segment besides the bytes of its rows, in elements (some 3 per ns and CTA): its
    # first loads, and the factor values of its columns. A row of few columns costs as much as one of 192, of 256 or 384
    # where accesses take 8 or 4 bytes: a group's threads go through all columns they might have. Shares by elements
    # alone left some CTAs with most of the segments: 8 x 1024^2 + 20 x 64^2 at rank 4 x 2 175 us per pass, 78 now, 84 by the
    # launches apart; ResNet-18 at 2 x 2 92, 82 and 84; 3 x 512x1024 at 2 x 2 43, 39 and 41.
    PANEL_START = (6144, 2304)   # and so many per factor column
    PANEL_ROW = {4: 192, 2: 256, 1: 384}

    def panel_costs(self, mats: Sequence[int], vec_widths: Sequence[int], columns: int) -> Tuple[np.ndarray, int]:
        """(what a row of each of the matrices costs at least, what a segment costs besides its rows) at so many factor columns."""
        return np.array([self.PANEL_ROW[int(vec_widths[mi])] for mi in mats]), self.PANEL_START[0] + self.PANEL_START[1] * columns

    def panel_pays(self, mats: Sequence[int], vec_widths: Sequence[int], columns: int, tc_flags: Sequence[bool], least: int) -> bool:
        """Is one pass over the matrices `mats` (and the launches apart for what is left) faster than the launches apart for
        all? `least`: elements that it needs in the best case. Measured as us per pass, accumulation included, launches apart /
        one pass, at rank 1 x 2, 2 x 2, 4 x 2, 8 x 1 (an odd number of half-iterations: per two passes, one of which ends on the
        Q side); over 90 random lists at 4 settings each it is on for half of them and 7 % faster there."""
        groups = [self.plan.groups[self.mats[mi][0]] for mi in mats]
        n, m = np.array([g.n for g in groups], dtype=np.int64), np.array([g.m for g in groups], dtype=np.int64)
        elems = int((n * m).sum())
        # Starts and narrow rows may cost an eighth: 320 x 64x640 (a quarter to a half) 142 / 136, 144 / 144, 164 / 167, 322 / 325;
        # 64 x 128x1024 (8, 12, 19 %) 65 / 58, 70 / 64, 82 / 79, 132 / 131; 4 x 24000x96 (double) 82 / 81, 90 / 95, 103 / 112, 175 / 184.
        # Starts of up to 16 rows are exempt, and elements of up to 8 rows count twice below: the launches apart pay as much for
        # tiles that are mostly empty (100 x 4x4096 67 / 46, 68 / 50, 99 / 78, 103 / 87).
        row, start = self.panel_costs(mats, vec_widths, columns)
        if 8 * int((n * np.maximum(m, row) + start * (n > 16)).sum()) > 9 * elems:
            return False
        tc_wide = int((n * m)[np.array([bool(tc_flags[mi]) for mi in mats]) & (m > 1024)].sum())
        if len(mats) < len(self.mats):
            # two more launches that fill the GPU badly: 8 x 2048^2 + 512x5000 227 / 236 ... 392 / 440, 4 x 4096^2 + 64x7000
            # 413 / 375 ... 718 / 690, + 512x7000 423 / 432 ... 728 / 750; 12 x 4096^2 + 512x7000 1127 / 1043 ... 1950 / 1912
            least *= 80 if 128 * (self.total_elems - elems) > elems else 28
        elif self.rt == 8 and 2 * tc_wide > elems:
            # the tensor cores make little of the product at rank 8, and rows of more than 1024 columns leave a CTA two
            # groups or one: 2 x 976x2048 at 8 x 1 86 / 93, 2 x 1952x2048 124 / 127, 2 x 2928x2048 164 / 163, 4 x 2048^2 210 / 200
            least *= 8
        elif columns > 4:
            # 6 x 512^2 44 / 48 at 4 x 2 (35 / 33 at 1 x 2, 39 / 39 at 2 x 2), 2 x 780x1024 45 / 47, 2 x 1024^2 47 / 47, 2 x 1220x1024 52 / 50
            least = least * 4 // 3
        return elems + int((n * m)[n <= 8].sum()) >= least

    def panel_segments(self, mats: Sequence[int], vec_widths: Sequence[int], rows_per_panel, row=0, start: int = 0) -> Tuple[np.ndarray, np.ndarray]:
        """Segments of whole rows of the matrices `mats` for the kernel that does the last product and the
        decompression in one pass, and the first segment of every CTA. Each CTA gets the same share of the work (`row`, `start`:
        see `panel_costs`), in quads of rows and in the order of the matrices. `rows_per_panel(m, rows)`: of a segment."""
        groups = [self.plan.groups[self.mats[mi][0]] for mi in mats]
        n, m = np.array([g.n for g in groups]), np.array([g.m for g in groups])
        quads, costs = (-(-n // 4)).astype(np.int64), (4 * np.maximum(m, row)).astype(np.int64)
        first_quad = np.concatenate([[0], np.cumsum(quads)])      # of every matrix, counted over all of them
        ctas = min(148, int(first_quad[-1]))
        bounds = np.zeros(ctas + 1, dtype=np.int64)   # where a CTA's share begins
        self._lib.psgd_panel_shares(quads.ctypes.data, costs.ctypes.data, len(mats), start, ctas, bounds.ctypes.data)
        cuts = np.union1d(bounds, first_quad)
        of = np.searchsorted(first_quad, cuts[:-1], side="right") - 1
        segs = np.zeros(len(cuts) - 1, dtype=layout.TILE_DTYPE)
        segs["mat"], segs["vec"] = np.array(mats)[of], np.array(vec_widths)[np.array(mats)[of]]
        segs["row0"], segs["cols"], segs["nsplit"] = 4 * (cuts[:-1] - first_quad[of]), m[of], 1
        segs["rows"] = np.minimum(4 * (cuts[1:] - first_quad[of]), n[of]) - segs["row0"]
        segs["split"] = [rows_per_panel(c, r) for c, r in zip(segs["cols"].tolist(), segs["rows"].tolist())]
        return segs, np.searchsorted(cuts, bounds).astype(np.int32)

    def orth_units(self, side: str, chunk_rows: int) -> Tuple[np.ndarray, np.ndarray]:
        """Units (one per matrix; one per shape group at rank 1) and their row chunks of at most
        `chunk_rows` rows, which never straddle the sub-matrices of a rank-1 unit."""
        units, chunks = [], []
        mi = 0

        def add(base, length, nsub, r, first_mat):
            chunk0 = len(chunks)
            for sub in range(nsub):
                for r0 in range(0, length, chunk_rows):
                    chunks.append((len(units), sub, sub * length + r0, min(chunk_rows, length - r0)))
            units.append((base, length, nsub, r, first_mat, chunk0, len(chunks) - chunk0, 0))

        for g in self.plan.groups:
            length = g.n if side == "p" else g.m
            base = g.p_offset if side == "p" else g.q_offset
            if g.r == 1:
                add(base, length, g.batch, 1, mi)
            else:
                for b in range(g.batch):
                    add(base + b * length * g.r, length, 1, g.r, mi + b)
            mi += g.batch
        return np.array(units, dtype=layout.ORTH_UNIT_DTYPE), np.array(chunks, dtype=layout.ORTH_CHUNK_DTYPE)


class _Recordable:
    """What an object keeps about launches that read its tables: the stream of the last ones that were not
    recorded, and, for recorded ones, the recording and what it refers to."""

    _stream: Optional[ctypes.c_void_p] = None
    recorded_in = 0

    def _owned(self) -> tuple:
        raise NotImplementedError

    @contextlib.contextmanager
    def _being_recorded(self, stream: ctypes.c_void_p):
        if not hasattr(self, "_kept"):
            self._kept: dict = {}
        keep_with_graph(self._kept, *self._owned())
        self.recorded_in = native.capture_id(stream)
        before = self._stream
        try:
            yield
        finally:
            self._stream = before


class _Tape:
    """Launches written down by the library, to be made again by one call of it. Only their arguments are kept."""

    def __init__(self, lib, body):
        self._lib, self._launches = lib, None
        try:   # (an interrupt may come anywhere)
            self._launches = lib.psgd_tape_begin()
            body()
        finally:
            self.count = lib.psgd_tape_end()

    def __del__(self):
        self._lib.psgd_tape_free(self._launches)

    def __call__(self, stream: ctypes.c_void_p) -> None:
        code = self._lib.psgd_tape_replay(self._launches, stream)
        if code != 0:
            native.check(code, "psgd_tape_replay")


class NativeCompressor(_Recordable):
    """Runs `BasicPowerSGD.aggregate` on the GPU with the in-tree kernels."""

    # sides whose factors may be orthonormalised in one launch, a cluster per unit, and those of them where that is the rule
    _orth_clusters: Dict[str, bool] = {}
    _orth_by_rule: Dict[str, bool] = {}

    # Elements of a list from which on one launch is the rule. It pays below as well: a replayed step gains 3 to 4 us of 31 to 35 (two
    # launches / one: 784x256 at rank 2 34.8 / 30.7). But lists that small have reported a fixed number of launches (`launches`), which the tests
    # hold: seven for 254 164 elements at two half-iterations. The line lies above that one, and an
    # orthonormalisation behind one ahead of time (`begin_step`) does not heed it: a recorded training step 101.2 / 98.2 us.
    ORTH_CLUSTER_ELEMS = 1 << 18

    def __init__(self, core):
        # the owner holds this object, not the other way round: both then go when the owner is dropped, and
        # not whenever the cycle collector runs - which may be in the middle of a CUDA-graph capture,
        # where giving back pinned memory ends the capture with an error
        self.core = weakref.proxy(core)
        self.lib = native.lib()
        self.device = core.device
        self.plan = core.plan
        self.tiles = TilePlan(core.plan, self.lib)
        self.T = core.config.num_iters_per_step
        self.tiles.fin_tc_ok = (
            self.T * self.tiles.max_r <= self.lib.psgd_finalize_tc_max_k()
            and os.environ.get("PSGD_B200_FINALIZE", "ffma") == "tc"
        )
        if self.T > layout.MAX_HIST:
            raise ValueError(f"num_iters_per_step {self.T} exceeds the compiled maximum {layout.MAX_HIST}")
        # finalize strips: as tall as the factor panels allow in shared memory, but short enough
        # that a small model still spreads over ~3 strips per SM (a strip costs its panels and one start).
        # 12 / 6 / 3 strips per SM, us per launch without the optimizer step, data in L2: ResNet-18 at 2 x 2 columns
        # 28.4 / 22.9 / 23.6, 2 x 2048^2 at 4 x 2 20.0 / 17.3 / 17.4, 17000x650 at 4 x 2 35.4 / 29.2 / 29.4, 8 x 1024x1001
        # at 16 x 2 45.7 / 35.1 / 31.0, 4 x 1024^2 at 8 x 1 and 3 x 1001x777 + 2 x 515x2049 at 3 x 3 alike within 8 %;
        # ResNet-18's recorded step 131 / 121.5 / 120.
        strip_cap = int(self.lib.psgd_finalize_strip_rows(self.T * self.tiles.max_r, 1 if world_size() == 1 else 0))
        want = self.tiles.total_elems // (128 * 148 * 3)
        self.tiles.fin_rows = max(32, min(strip_cap, want // 32 * 32))
        nm = len(self.tiles.mats)
        cap = max(self.plan.p_total, self.plan.q_total, 1)
        f32 = dict(device=self.device, dtype=torch.float32)
        self.h_in = [torch.zeros(cap, **f32) for _ in range(self.T)]
        self.h_loc = [torch.zeros(cap, **f32) for _ in range(self.T)]
        self.h_sum = [torch.zeros(cap, **f32) for _ in range(self.T)]
        self.cmat = [[torch.zeros(nm * layout.CMAT_STRIDE, **f32) for _ in range(t)] for t in range(self.T)]
        rt = int(self.lib.psgd_orth_template_rank(self.tiles.max_r))
        self.units, self.chunks, self.n_units, self.n_chunks = {}, {}, {}, {}
        self._orth_clusters, self._orth_by_rule = {}, {}
        for s in ("p", "q"):
            longest = max(((g.n if s == "p" else g.m) * (g.batch if g.r == 1 else 1) for g in self.plan.groups), default=1)
            units, chunks = self.tiles.orth_units(s, int(self.lib.psgd_orth_chunk_rows(self.tiles.max_r, longest)))
            self.units[s], self.chunks[s] = _to_device(units, self.device), _to_device(chunks, self.device)
            self.n_units[s], self.n_chunks[s] = len(units), len(chunks)
            if world_size() == 1:
                members = max((g.batch for g in self.plan.groups if g.r == 1), default=1)
                rows = sum((g.n if s == "p" else g.m) * g.batch for g in self.plan.groups)
                self._orth_clusters[s] = bool(self.lib.psgd_orth_takes_clusters(self.tiles.max_r, longest, members, max(self.T - 1, 0), len(units), rows))
                self._orth_by_rule[s] = self._orth_clusters[s] and self.tiles.total_elems >= self.ORTH_CLUSTER_ELEMS
        # scratch of the orthonormalisation: partial sums per chunk; per unit (`_orth_rinv`) the leading
        # rows of the factor as they came in, which R falls back on when a column has to be replaced
        part_doubles = int(self.lib.psgd_orth_part_doubles(self.tiles.max_r, max(self.T - 1, 0)))
        max_units = max(max(self.n_units.values()), 1)
        self._orth_part = torch.zeros(max(max(self.n_chunks.values()), 1) * part_doubles, device=self.device, dtype=torch.float64)
        self._orth_rinv = torch.zeros(max_units * 2 * rt * rt, device=self.device, dtype=torch.float32)
        self._key = None
        self._tapes: Dict[Tuple, _Tape] = {}
        self._out_arena: Optional[torch.Tensor] = None
        self._hyper_dev = _to_device(self._default_hyper(), self.device)
        self.launches = 0  # kernels launched by the last aggregate()
        self._side_stream = torch.cuda.Stream(device=self.device)
        self._early = None  # (side, event) of an orthonormalisation issued by begin_step()
        self._early_launches = 0
        self._early_bucket: frozenset = frozenset()
        self._early_product_done = None  # event of a first product launched ahead for the early bucket
        # multi-GPU: factors are all-reduced by the product kernels themselves (peer pushes) plus
        # a small consumer kernel; PSGD_B200_COMM=nccl selects the library all-reduce instead
        self.comm = None
        if world_size() > 1 and os.environ.get("PSGD_B200_COMM", "p2p") == "p2p":
            from .parallel.symm import Channel, assert_same_on_all_ranks

            # a rank with another model, rank or iteration count would push factors of another
            # layout: find out now, with a message, instead of through a timeout later
            assert_same_on_all_ranks(
                (self.plan.signature(), int(core.config.rank), int(self.T)), "PowerSGD compression plan"
            )
            self.comm = Channel(cap)
        # status word of the bounded waits of the tensor-core and the one-pass kernels: mapped pinned host memory, so the
        # host can look at it every step without touching the GPU
        from .parallel.symm import StatusWord

        self._status = StatusWord()

    @staticmethod
    def _default_hyper() -> np.ndarray:
        h = np.zeros(1, dtype=layout.HYPER_DTYPE)
        h["grad_scale"] = 1.0
        h["one_minus_dampening"] = 1.0
        return h

    # -- descriptors -----------------------------------------------------------------------
    def _bind(
        self,
        grads: Sequence[torch.Tensor],
        params: Optional[Sequence[torch.Tensor]] = None,
        moms: Optional[Sequence[Optional[torch.Tensor]]] = None,
        hyper_index: Optional[Sequence[int]] = None,
        need_out: bool = True,
        outs: Optional[Sequence[torch.Tensor]] = None,
        finish: bool = False,
    ) -> None:
        """`outs`: caller-owned tensors (laid out like the gradients) that receive the averaged
        update instead of this object's own arena. `finish`: the caller's steps may end in the one-pass
        kernel (see `_half_iterations`); an object is always bound with the same."""
        key = (scan.addresses(grads), scan.addresses(params), scan.addresses(moms), need_out, scan.addresses(outs))
        if key == self._key:
            return
        for g in grads:
            if not is_dense(g) or g.dtype != torch.float32 or g.device != self.device:
                raise ValueError("native PowerSGD needs dense float32 gradients on its device")
        for name, others in (("parameters", params), ("momentum buffers", moms), ("outputs", outs)):
            for g, o in zip(grads, others or []):
                if o is not None and not same_layout(o, g):
                    raise ValueError(f"native PowerSGD needs {name} laid out like their gradients")
        if need_out and outs is None and self._out_arena is None:
            self._out_arena = torch.empty(self.tiles.total_elems, device=self.device, dtype=torch.float32)
        where = self.plan.locate()
        descs = np.zeros(len(self.tiles.mats), dtype=layout.MAT_DTYPE)
        vec = []
        out_views: List[Optional[torch.Tensor]] = [None] * len(grads)
        cursor = 0
        # output arena is laid out in compressed-list order so that views are plain slices
        out_offsets = []
        for g in grads:
            out_offsets.append(cursor)
            cursor += g.numel()
        for mi, (gi, pos, idx) in enumerate(self.tiles.mats):
            g = self.plan.groups[gi]
            d = descs[mi]
            d["grad"] = grads[idx].data_ptr()
            d["param"] = 0 if params is None else params[idx].data_ptr()
            d["mom"] = 0 if (moms is None or moms[idx] is None) else moms[idx].data_ptr()
            if need_out and outs is not None:
                out_views[idx] = outs[idx]
                d["out"] = outs[idx].data_ptr()
            elif need_out:
                view = self._out_arena[out_offsets[idx] : out_offsets[idx] + grads[idx].numel()]
                out_views[idx] = like_strided(view, grads[idx])
                d["out"] = view.data_ptr()
            d["n"], d["m"], d["r"] = g.n, g.m, g.r
            d["p_off"] = g.p_offset + pos * g.n * g.r
            d["q_off"] = g.q_offset + pos * g.m * g.r
            d["grp_p_off"], d["grp_p_len"] = g.p_offset, g.p_numel
            d["grp_q_off"], d["grp_q_len"] = g.q_offset, g.q_numel
            d["hyper"] = 0 if hyper_index is None else hyper_index[idx]
            d["index"] = mi
            ptrs = [int(d["grad"]), int(d["param"]), int(d["mom"]), int(d["out"])]
            # widest global access every row of the matrix (and of its companions) allows
            if g.m % 4 == 0 and all(p % 16 == 0 for p in ptrs):
                vec.append(4)
            elif g.m % 2 == 0 and all(p % 8 == 0 for p in ptrs):
                vec.append(2)
            else:
                vec.append(1)
        assert where is not None
        by_16 = sum(g.n * g.m for g, v in zip((self.plan.groups[gi] for gi, _pos, _idx in self.tiles.mats), vec) if v == 4)
        self._strip_flags = 4 if by_16 >= self.STRIPS_BY_16 * self.tiles.total_elems else 0
        self._mats_dev = _to_device(descs, self.device)
        # tensor-core (TMA + tcgen05) path: matrices TMA can address and that are worth it
        mode = os.environ.get("PSGD_B200_GEMM", "auto")
        hbm_bound = self.tiles.total_elems * 4 > (96 << 20)
        tc = []
        maps = np.zeros((len(self.tiles.mats), 256), dtype=np.uint8)
        for mi, (gi, _pos, idx) in enumerate(self.tiles.mats):
            g = self.plan.groups[gi]
            ok = vec[mi] == 4 and g.n >= 128 and g.m >= 128 and mode != "ffma"
            ok = ok and (mode == "tc" or hbm_bound or self.tiles.max_r >= 8)
            if ok:
                buf = (ctypes.c_ubyte * 256)()
                code = self.lib.psgd_tma_encode_matrix(buf, ctypes.c_void_p(grads[idx].data_ptr()), g.n, g.m)
                native.check(code, "psgd_tma_encode_matrix")
                maps[mi] = np.frombuffer(buf, dtype=np.uint8)
            tc.append(bool(ok))
        self._maps_dev = _to_device(maps, self.device)
        self._tc_split = os.environ.get("PSGD_B200_TC_PRECISION", "split") != "tf32"
        self.uses_tensor_cores = any(tc)
        # compressed-list positions whose products run on the tensor-core kernels (one launch per
        # half-iteration for all of them; they are not split into an early and a late bucket)
        self.tensor_core_positions = frozenset(idx for (_gi, _pos, idx), flag in zip(self.tiles.mats, tc) if flag)
        tile_arrays = self.tiles.build(vec, tc)
        self._tile_arrays = tile_arrays
        self._tiles_dev: Dict[str, Dict[int, Tuple[torch.Tensor, int]]] = {}
        for name, by_vec in tile_arrays.items():
            self._tiles_dev[name] = {
                v: (_to_device(a, self.device) if len(a) else None, len(a)) for v, a in by_vec.items()
            }
        self._panel = None
        if finish:
            self._plan_panels(vec, [grads[idx].data_ptr() for _gi, _pos, idx in self.tiles.mats], mode, tc)
        self._split_tile_lists()
        self._partial = torch.empty(self.tiles.partial_floats, device=self.device, dtype=torch.float32)
        self._partial_tc = torch.empty(self.tiles.partial_tc_floats, device=self.device, dtype=torch.float32)
        with outside_capture(self.device):   # zero between launches: every launch leaves them so
            self._tickets = torch.zeros(self.tiles.n_tickets, device=self.device, dtype=torch.int32)
        self._out_views = out_views
        self._tapes.clear()
        self._key = key

    # Share of elements accessed by 16 bytes from which on the decompression takes the form for those (csrc/finalize.cu, ROWS):
    # 94 % loses 3 % at 16 factor columns, 98 % loses nothing.
    STRIPS_BY_16 = 31 / 32

    # Elements from which on a step may end in the one-pass kernel (0: wherever it can), see `panel_pays`. At rank 1 x 2, launches
    # apart / one pass: 2 x 512^2 30.7 / 30.8, 2 x 512x1024 33.8 / 31.6, 2 x 780x1024 37 / 33, 2 x 1952x1024 43 / 37, 4 x 2048^2 114 / 92 us.
    PANEL_ELEMS = 3 << 19

    def _plan_panels(self, vec: Sequence[int], addresses: Sequence[int], mode: str, tc: Sequence[bool]) -> None:
        """Which matrices finish a step whose last basis is on the Q side in one pass (csrc/panel.cu), and the tile
        lists of the others. One worker, no optimizer step, no product kernel asked for by name."""
        if world_size() != 1 or mode != "auto" or self.tiles.fin_tc_ok or self.tiles.total_elems < self.PANEL_ELEMS:
            return
        known: Dict[Tuple[int, int], int] = {}

        def rows(m: int, n: int) -> int:
            if (m, n) not in known:
                known[m, n] = int(self.lib.psgd_panel_rows(self.tiles.max_r, self.T, m, n))
            return known[m, n]

        groups = [self.plan.groups[gi] for gi, _pos, _idx in self.tiles.mats]
        mats = [mi for mi, (g, at) in enumerate(zip(groups, addresses)) if at % 16 == 0 and rows(g.m, g.n) > 0]
        columns = self.tiles.rt * self.T
        if not mats or (self.PANEL_ELEMS and not self.tiles.panel_pays(mats, vec, columns, tc, self.PANEL_ELEMS)):
            return
        segs, starts = self.tiles.panel_segments(mats, vec, rows, *self.tiles.panel_costs(mats, vec, columns))
        table = _to_device(np.concatenate([segs.view(np.uint8), starts.view(np.uint8)]), self.device)
        self._panel = (table, segs.nbytes, len(starts) - 1)
        for name in ("nn", "fin"):
            for key in ("f", "tc"):
                arr = self._tile_arrays[name][key]
                rest = arr[~np.isin(arr["mat"], mats)] if len(arr) and len(mats) < len(groups) else arr[:0]
                self._tiles_dev[name][key + "_rest"] = (_to_device(rest, self.device) if len(rest) else None, len(rest))

    # -- early bucket ---------------------------------------------------------------------
    def set_early_bucket(self, compressed_indices: Sequence[int]) -> None:
        """Compressed tensors (positions in the compressed list) whose gradients are complete
        early in backward: the first product of a step can be launched for them from a
        post-accumulate hook, on a side stream, while backward is still running for the rest."""
        self._early_bucket = frozenset(int(i) for i in compressed_indices)
        if self._key is not None:
            self._split_tile_lists()

    def _split_tile_lists(self) -> None:
        """Product tile lists of the early bucket ("fA") and of everything else ("fB")."""
        early_mats = [mi for mi, (_gi, _pos, idx) in enumerate(self.tiles.mats) if idx in self._early_bucket]
        for name in ("nt", "nn"):
            if not early_mats:
                self._tiles_dev[name].update(fA=(None, 0), fB=self._tiles_dev[name]["f"])
                continue
            arr = self._tile_arrays[name]["f"]
            mask = np.isin(arr["mat"], early_mats) if len(arr) else np.zeros(0, dtype=bool)
            for key, sub in (("fA", arr[mask]), ("fB", arr[~mask])):
                self._tiles_dev[name][key] = (_to_device(np.ascontiguousarray(sub), self.device) if len(sub) else None, len(sub))

    def early_product(self) -> bool:
        """Launch the first product of the coming step for the early bucket NOW, on the side
        stream (after the orthonormalisation `begin_step` issued there). Returns False when there
        is nothing to launch early. `_half_iterations` then only launches the rest and joins."""
        if not self._early_bucket or self._early is None or self._key is None:
            return False
        core = self.core
        left = (core.step_counter * self.T) % 2 == 0
        if self._early[0] != ("p" if left else "q"):
            return False
        name = "nt" if left else "nn"
        if self._tiles_dev[name]["fA"][1] == 0:
            return False
        state_out = core._qs_buffer if left else core._ps_buffer
        fork = torch.cuda.Event()
        fork.record(torch.cuda.current_stream())
        self._side_stream.wait_event(fork)
        with torch.cuda.stream(self._side_stream):
            before = self.launches
            self._gemm(left, self.h_in[0], self.h_loc[0], [], self.cmat[0], state_out if world_size() == 1 else None, part="early")
            self._early_launches += self.launches - before
            done = torch.cuda.Event()
            done.record(self._side_stream)
        self._early_product_done = done
        return True

    # -- launches --------------------------------------------------------------------------
    def _call(self, name: str, *args) -> None:
        """One launch of the library on the current stream, counted."""
        fn = getattr(self.lib, name)
        self._stream = _stream_ptr()
        native.check(fn(*args, self._stream), name)
        launched = 2 if name == "psgd_orth_launch" and not args[-1] & 4 else 1   # orthonormalisation: Gram matrices, then their use
        self.launches += launched

    def _taped(self, key: Tuple, body, inside: bool = False) -> None:
        """Run `body`, which issues the launches of a step; from the second step of its kind on repeat
        the same calls with the arguments they had, without working them out again (an eager loop over
        a small model spends most of its step there). `key`: whatever the arguments depend on beyond
        the bound tensors; a new binding drops all tapes. Only where a step is nothing but launches on
        one stream: one worker, nothing launched ahead, no phase timing."""
        stream = _stream_ptr()
        if stream and not inside and is_recorded(stream):   # (0, the default stream: never)
            with self._being_recorded(stream):
                self._taped(key, body, inside=True)
            return
        plain = (world_size() == 1 and self.comm is None and self._early is None and self._early_product_done is None
                 and not _Range.enabled and _Range.events is None)
        if not plain:
            body()
            return
        key = key + (self.core._ps_buffer.data_ptr(), self.core._qs_buffer.data_ptr())
        tape = self._tapes.get(key)
        if tape is None:
            before = self.launches
            tape = _Tape(self.lib, body)
            if tape.count == self.launches - before:   # (all of them went through the library's one way of launching)
                if len(self._tapes) >= 16:   # recordings with tables of their own bring keys of their own
                    self._tapes.clear()
                self._tapes[key] = tape
            return
        self._stream = stream
        tape(stream)
        self.launches += tape.count

    def _owned(self) -> tuple:
        """Everything a step addresses besides the caller's tensors; the next binding replaces the tables and
        the scratch."""
        return (
            self._mats_dev, self._maps_dev, *(t for lists in self._tiles_dev.values() for t, _count in lists.values()),
            self._panel, self._partial, self._partial_tc, self._tickets, self._out_arena, self._hyper_dev, self._status,
            self.units, self.chunks, self._orth_part, self._orth_rinv, self.h_in, self.h_loc, self.h_sum, self.cmat,
            self.core._ps_buffer, self.core._qs_buffer,
        )

    # -- phases ----------------------------------------------------------------------------
    def _orth(self, side: str, x: torch.Tensor, copy_to: torch.Tensor, prev: List[torch.Tensor], cm: List[torch.Tensor],
              gather_to: Optional[torch.Tensor] = None, early: bool = False, same: bool = False,
              clusters: Optional[bool] = None):
        """Orthonormalise `x` in place (mirrored into `copy_to`). With `gather_to`, `x` is first
        filled with the sum over workers of the factor the previous product pushed (the sum is
        also written to `gather_to`): the launch is the consumer of the in-kernel all-reduce.
        `early`: see `_chained`. `same`: the last factor in `prev` is a copy of `x` as it comes in. `clusters`: one
        launch where it can be (True), never (False), by the rule (None)."""
        clusters = gather_to is None and clusters is not False and (self._orth_clusters if clusters else self._orth_by_rule).get(side, False)
        self._call(
            "psgd_orth_launch",
            _ptr(self.units[side]),
            self.n_units[side],
            _ptr(self.chunks[side]),
            self.n_chunks[side],
            self.tiles.max_r,
            _ptr(x),
            _ptr(copy_to),
            len(prev),
            ctypes.cast(_ptr_array(prev), ctypes.c_void_p),
            ctypes.cast(_ptr_array(cm), ctypes.c_void_p),
            _ptr(self._orth_part),
            _ptr(self._orth_rinv),
            self.comm.ptr if gather_to is not None else ctypes.c_void_p(0),
            _ptr(gather_to),
            (1 if early else 0) | ((12 if same else 4) if clusters else 2 if self._chained() else 0),   # the second launch follows the first
        )

    def _chained(self) -> bool:
        """May a launch whose direct predecessor in the stream is a launch of the same step start
        before that one has ended (csrc/psgd_common.cuh, psgd_launch)? One worker only: what several
        workers exchange inside the kernels keeps the plain stream order."""
        return self.comm is None and world_size() == 1

    def _gemm(self, transposed: bool, fin: torch.Tensor, fout: torch.Tensor, corr_fac, corr_c,
              fout2: Optional[torch.Tensor] = None, part: str = "all", early: bool = False):
        """`part`: "all", or one half of a split launch - "early" (the CUDA-core tiles of the
        matrices in the early bucket) / "late" (everything else); see `set_early_bucket` -, or
        "rest" (what the panel kernel leaves). `early`: see `_chained`."""
        name = "nt" if transposed else "nn"
        form = (1 if transposed else 0) | (2 if early else 0)
        tiles, count = self._tiles_dev[name]["tc_rest" if part == "rest" else "tc"]
        if count and part != "early":
            self._call(
                "psgd_gemm_tc_launch",
                form,
                1 if self._tc_split else 0,
                self.tiles.max_r,
                _ptr(self._mats_dev),
                _ptr(tiles),
                count,
                _ptr(self._maps_dev),
                _ptr(fin),
                _ptr(fout),
                _ptr(fout2),
                len(corr_fac),
                ctypes.cast(_ptr_array(corr_fac), ctypes.c_void_p),
                ctypes.cast(_ptr_array(corr_c), ctypes.c_void_p),
                _ptr(self._partial_tc),
                _ptr(self._tickets),
                self.comm.ptr if self.comm is not None else ctypes.c_void_p(0),
                self._status.dev_ptr,
            )
        tiles, count = self._tiles_dev[name][{"all": "f", "early": "fA", "late": "fB", "rest": "f_rest"}[part]]
        if count:
            self._call(
                "psgd_gemm_ffma_launch",
                form,
                self.tiles.max_r,
                _ptr(self._mats_dev),
                _ptr(tiles),
                count,
                _ptr(fin),
                _ptr(fout),
                _ptr(fout2),
                len(corr_fac),
                ctypes.cast(_ptr_array(corr_fac), ctypes.c_void_p),
                ctypes.cast(_ptr_array(corr_c), ctypes.c_void_p),
                _ptr(self._partial),
                _ptr(self._tickets),
                self.comm.ptr if self.comm is not None else ctypes.c_void_p(0),
            )

    def _gathers_in_finalize(self) -> bool:
        """Multi-GPU: can the decompression launch gather the last factor from the channel itself?
        Only the strip kernel does, and only when it is the sole decompression launch."""
        if self.comm is None or world_size() == 1:
            return False
        if self._tiles_dev["fin"]["tc"][1]:
            return False
        return bool(self.lib.psgd_finalize_uses_strip(self.T, self.tiles.max_r, self.tiles.fin_rows, 0))

    def _finalize(self, sides: List[bool], fused_sgd: bool, workers: int, gather_state: Optional[torch.Tensor] = None,
                  flags: int = 0, early: bool = False, rest: bool = False):
        """`rest`: only the matrices that the panel kernel leaves. `gather_state`: the warm-start buffer that receives the summed factor of the last
        half-iteration when this launch is also its consumer (see `_gathers_in_finalize`).
        `flags`: residual options of the strip / general kernels (csrc/finalize.cu, FinalizeArgs).
        `early`: see `_chained`."""
        if flags and self._tiles_dev["fin"]["tc"][1]:
            raise ValueError("residual options are not available with the tensor-core decompression kernel")
        lloc, rloc, lsum, rsum = [], [], [], []
        for t, left in enumerate(sides):
            if left:
                lloc.append(self.h_in[t]); lsum.append(self.h_in[t])
                rloc.append(self.h_loc[t]); rsum.append(self.h_sum[t])
            else:
                rloc.append(self.h_in[t]); rsum.append(self.h_in[t])
                lloc.append(self.h_loc[t]); lsum.append(self.h_sum[t])
        tiles, count = self._tiles_dev["fin"]["tc_rest" if rest else "tc"]
        if count:
            self._call(
                "psgd_finalize_tc_launch",
                _ptr(self._mats_dev),
                _ptr(tiles),
                count,
                _ptr(self._maps_dev),
                _ptr(self._hyper_dev),
                len(sides),
                self.tiles.max_r,
                ctypes.cast(_ptr_array(lloc), ctypes.c_void_p),
                ctypes.cast(_ptr_array(rloc), ctypes.c_void_p),
                ctypes.cast(_ptr_array(lsum), ctypes.c_void_p),
                ctypes.cast(_ptr_array(rsum), ctypes.c_void_p),
                1.0 / workers,
                1 if fused_sgd else 0,
                self._status.dev_ptr,
            )
        tiles, count = self._tiles_dev["fin"]["f_rest" if rest else "f"]
        if count:
            gather = gather_state is not None
            self._call(
                "psgd_finalize_launch",
                _ptr(self._mats_dev),
                _ptr(tiles),
                count,
                self.tiles.fin_rows,
                self.tiles.max_r,
                _ptr(self._hyper_dev),
                len(sides),
                ctypes.cast(_ptr_array(lloc), ctypes.c_void_p),
                ctypes.cast(_ptr_array(rloc), ctypes.c_void_p),
                ctypes.cast(_ptr_array(lsum), ctypes.c_void_p),
                ctypes.cast(_ptr_array(rsum), ctypes.c_void_p),
                1.0 / workers,
                1 if fused_sgd else 0,
                self.comm.ptr if gather else ctypes.c_void_p(0),
                0 if sides[-1] else 1,  # last half-iteration left: the fresh (summed) factor is the right one
                _ptr(self.h_sum[len(sides) - 1]) if gather else ctypes.c_void_p(0),
                _ptr(gather_state) if gather else ctypes.c_void_p(0),
                int(flags) | self._strip_flags,
                1.0,
                int(early and not self._tiles_dev["fin"]["tc"][1]),
            )

    def _finish_panels(self, sides: List[bool], state_out: torch.Tensor, early: bool) -> None:
        """The last half-iteration (basis on the Q side) and the decompression of the matrices that take one
        pass for both. `early`: see `_chained`."""
        last = len(sides) - 1
        left = [self.h_in[t] if sides[t] else self.h_loc[t] for t in range(last)]
        right = [self.h_loc[t] if sides[t] else self.h_in[t] for t in range(last)]
        table, segs_bytes, ctas = self._panel
        self._call(
            "psgd_panel_launch",
            _ptr(self._mats_dev), _ptr(table), ctypes.c_void_p(table.data_ptr() + segs_bytes), ctas, self.tiles.max_r, len(sides),
            _ptr(self.h_in[last]), _ptr(self.h_loc[last]), _ptr(state_out),
            ctypes.cast(_ptr_array(left), ctypes.c_void_p), ctypes.cast(_ptr_array(right), ctypes.c_void_p),
            ctypes.cast(_ptr_array(self.cmat[last]), ctypes.c_void_p), self._status.dev_ptr, int(early),
        )

    def _half_iterations(self, finish: bool = False):
        """Runs the T half-iterations. Returns (sides, pending): `pending` is the warm-start buffer
        whose summed factor the decompression launch still has to gather, or None. `_follows` says
        whether the last thing put on the stream was a launch of the step (see `_chained`), `_finished` whether
        the last one was also the decompression of the matrices that the panel kernel takes, which `finish` allows."""
        core = self.core
        workers = world_size()
        p2p = workers > 1 and self.comm is not None
        defer_last = p2p and self._gathers_in_finalize()
        sides: List[bool] = []
        pending: Optional[torch.Tensor] = None   # state buffer whose sum is still in the channel's slots
        chained, self._follows, self._finished = self._chained(), False, False
        ahead = self._early is not None
        for t in range(self.T):
            left = (core.step_counter * self.T + t) % 2 == 0
            sides.append(left)
            side = "p" if left else "q"
            state_in = core._ps_buffer if left else core._qs_buffer
            state_out = core._qs_buffer if left else core._ps_buffer
            # earlier LOCAL factors on the input side (cross products) and on the output side (corrections)
            same, other = [], []
            for i in range(t):
                in_side_i = self.h_in[i] if sides[i] == left else self.h_loc[i]
                out_side_i = self.h_loc[i] if sides[i] == left else self.h_in[i]
                same.append(in_side_i)
                other.append(out_side_i)
            with _Range(f"psgd.iter{t}.orth"):
                gather_to = None
                if pending is not None:
                    # the basis of this half-iteration IS the factor the previous product pushed
                    assert pending is state_in
                    gather_to, pending = self.h_sum[t - 1], None
                if t == 0 and self._early is not None:
                    # the first basis was orthonormalised on the side stream while forward / backward ran
                    early_side, event = self._early
                    self._early = None
                    torch.cuda.current_stream().wait_event(event)
                    if early_side != side:  # state changed under us (e.g. a checkpoint was loaded): redo
                        self._orth(side, state_in, self.h_in[t], same, self.cmat[t])
                else:
                    # the first launch of a step waits for all work before it (gradients, parameters)
                    self._orth(side, state_in, self.h_in[t], same, self.cmat[t], gather_to, early=self._follows,
                               same=t > 0 and workers == 1, clusters=ahead or None)
                    self._follows = chained
            with _Range(f"psgd.iter{t}.product"):
                # one worker: the product is final, so the kernel also writes the warm-start buffer
                part = "all"
                if t == 0 and self._early_product_done is not None:
                    part = "late"  # the early bucket's tiles were launched during backward
                elif finish and t == self.T - 1 and not left and self._panel is not None:
                    part, self._finished = "rest", True
                self._gemm(left, self.h_in[t], self.h_loc[t], other, self.cmat[t], state_out if workers == 1 else None, part=part,
                           early=self._follows)
                if part == "rest":
                    self._finish_panels(sides, state_out, early=self._follows)
                self._follows = chained
                if part == "late":
                    torch.cuda.current_stream().wait_event(self._early_product_done)
                    self._early_product_done = None
                    self._follows = False
            total = state_out.numel()
            with _Range(f"psgd.iter{t}.reduce"):
                if p2p and (t < self.T - 1 or defer_last):
                    pending = state_out  # gathered by the next consumer of that factor
                elif p2p:
                    code = self.lib.psgd_factor_reduce_launch(
                        self.comm.ptr, ctypes.c_longlong(total), _ptr(self.h_sum[t]), _ptr(state_out), _stream_ptr()
                    )
                    native.check(code, "psgd_factor_reduce_launch")
                    self.launches += 1
                elif workers > 1:
                    self.h_sum[t][:total].copy_(self.h_loc[t][:total])
                    self._allreduce_sum(self.h_sum[t][:total])
                    state_out.copy_(self.h_sum[t][:total])
        return sides, pending

    def _allreduce_sum(self, flat: torch.Tensor) -> None:
        dist.all_reduce(flat)

    def begin_step(self) -> None:
        """Orthonormalise the basis of the first half-iteration NOW, on a side stream.

        That basis only depends on the factors left by the previous step, not on the gradients
        about to be computed, so the launch overlaps with forward / backward; `aggregate` then
        waits on an event instead of launching it. Captured in a CUDA graph this is a parallel
        branch of the step."""
        if self._early is not None:
            return
        core = self.core
        left = (core.step_counter * self.T) % 2 == 0
        side = "p" if left else "q"
        state_in = core._ps_buffer if left else core._qs_buffer
        main = torch.cuda.current_stream()
        fork = torch.cuda.Event()
        fork.record(main)
        self._side_stream.wait_event(fork)
        with torch.cuda.stream(self._side_stream):
            before = self.launches
            # two launches: as the first node of a graph's side branch a launch with clusters delays the whole graph, 101 -> 107 us
            # for a recorded step of a small perceptron, and there is nothing to gain off the critical path
            self._orth(side, state_in, self.h_in[0], [], self.cmat[0], clusters=False)
            self._early_launches = self.launches - before  # counted with the step that uses them
            done = torch.cuda.Event()
            done.record(self._side_stream)
        self._early = (side, done)

    def close(self) -> None:
        """Release the peer mappings and the symmetric arena (collective across ranks)."""
        if self.comm is not None:
            self.comm.close()
            self.comm = None

    def check(self) -> None:
        """Raise `PowerSGDCommTimeout` if a bounded device-side wait of an EARLIER launch gave up
        (a peer that never pushed, copies into shared memory or tensor-core work that never ended). Plain host reads of
        mapped pinned words: no synchronisation, cheap enough for every step."""
        if self.comm is not None:
            self.comm.check()
        self._status.check("a wait inside a product, decompression or one-pass kernel")

    # -- public ----------------------------------------------------------------------------
    def aggregate(self, gradients: List[torch.Tensor]) -> List[torch.Tensor]:
        self.check()
        self.launches = self._early_launches if self._early is not None else 0
        self._bind(gradients, finish=True)
        self._taped((self._first_left(), False), lambda: self._step(fused_sgd=False))
        return list(self._out_views)

    def _first_left(self) -> bool:
        return (self.core.step_counter * self.T) % 2 == 0

    def _step(self, fused_sgd: bool) -> None:
        workers = world_size()
        if workers == 1:
            saved = self.h_sum
            self.h_sum = self.h_loc
        try:
            sides, pending = self._half_iterations(finish=not fused_sgd)
            with _Range("psgd.finalize+sgd" if fused_sgd else "psgd.finalize"):
                self._finalize(sides, fused_sgd=fused_sgd, workers=workers, gather_state=pending, early=self._follows,
                               rest=self._finished)
        finally:
            if workers == 1:
                self.h_sum = saved

    def aggregate_and_step(
        self,
        gradients: List[torch.Tensor],
        params: List[torch.Tensor],
        moms: List[Optional[torch.Tensor]],
        hyper_index: List[int],
        hyper_dev: torch.Tensor,
    ) -> None:
        """Same as `aggregate`, but applies SGD to `params` inside the last kernel instead of
        materialising the averaged gradients."""
        self.check()
        self.launches = self._early_launches if self._early is not None else 0
        self._bind(gradients, params, moms, hyper_index, need_out=False)
        keep = self._hyper_dev
        self._hyper_dev = hyper_dev
        try:
            self._taped((self._first_left(), True, hyper_dev.data_ptr()), lambda: self._step(fused_sgd=True))
        finally:
            self._hyper_dev = keep


class NativeFlatAllReduce(_Recordable):
    """Mean of a list of float32 tensors through one flat buffer, with the packing, the 1/W
    scale, the zeroing of the inputs and (optionally) the SGD update done by one multi-tensor
    kernel on each side of the collective."""

    # one-shot pushes send (W-1) copies of the buffer: right for the small per-step buffers
    # (latency of one hop). Larger ones (whole models: the plain all-reduce aggregator, the
    # un-compressed warm-up phase) go two-shot: reduce-scatter + all-gather through peer stores,
    # 2 (W-1)/W copies. Beyond the arena limit the library ring takes over (eager only).
    ONE_SHOT_LIMIT_FLOATS = 1 << 18
    P2P_ARENA_LIMIT_BYTES = 8 << 30

    def __init__(self):
        self.lib = native.lib()
        self._key = None
        self.launches = 0
        self.comm = None
        self.path = "local"
        self.n_pad = 0
        self._bulk_layout = None
        self._pushed = False  # one-shot path: this step's pack + push already left with another launch
        self._keep_inputs = False
        self._nvls = None     # in-switch all-reduce object (parallel/nvls.py)
        self._nvls_failed = False
        self._tapes: Dict[Tuple, _Tape] = {}   # of one worker's launch, see NativeCompressor._taped

    def check(self) -> None:
        """Raise `PowerSGDCommTimeout` if a bounded wait of an earlier launch gave up."""
        if self.comm is not None:
            self.comm.check()
        if self._nvls is not None:
            self._nvls.check()

    def _bind(self, grads, params=None, moms=None, hyper_index=None, need_out=True, outs=None):
        key = (scan.addresses(grads), scan.addresses(params), scan.addresses(moms), need_out, scan.addresses(outs))
        if key == self._key:
            return
        device = grads[0].device
        # every tensor starts at a multiple of four floats in the flat buffer (16-byte accesses)
        total = sum(-(-g.numel() // 4) * 4 for g in grads)
        self._out = torch.empty(total, device=device, dtype=torch.float32) if (need_out and outs is None) else None
        items = np.zeros(len(grads), dtype=layout.FLAT_DTYPE)
        per_block = self.lib.psgd_flat_block_elems()
        block_item, block_first = [], []
        views, cursor = [], 0
        for i, g in enumerate(grads):
            if not is_dense(g) or g.dtype != torch.float32:
                raise ValueError("native flat all-reduce needs dense float32 tensors")
            for o in ((params[i] if params is not None else None), (moms[i] if moms is not None else None),
                      (outs[i] if outs is not None else None)):
                if o is not None and not same_layout(o, g):
                    raise ValueError("native flat all-reduce needs parameters, momentum buffers and outputs laid out like the gradients")
            it = items[i]
            it["grad"] = g.data_ptr()
            it["param"] = 0 if params is None else params[i].data_ptr()
            it["mom"] = 0 if (moms is None or moms[i] is None) else moms[i].data_ptr()
            if need_out and outs is not None:
                views.append(outs[i])
                it["out"] = outs[i].data_ptr()
            elif need_out:
                v = self._out[cursor : cursor + g.numel()]
                views.append(like_strided(v, g))
                it["out"] = v.data_ptr()
            it["numel"] = g.numel()
            it["flat_off"] = cursor
            it["hyper"] = 0 if hyper_index is None else hyper_index[i]
            for first in range(0, g.numel(), per_block):
                block_item.append(i)
                block_first.append(first)
            cursor += -(-g.numel() // 4) * 4
        pointers = [int(items[name][i]) for name in ("grad", "param", "mom", "out") for i in range(len(grads))]
        self._vec = 1 if all(ptr % 16 == 0 for ptr in pointers) else 0
        self._items_dev = _to_device(items, device)
        self._items_host = items
        self._block_item = _to_device(np.asarray(block_item, dtype=np.int32), device)
        self._block_first = _to_device(np.asarray(block_first, dtype=np.int32), device)
        self._nblocks = len(block_item)
        self._views = views
        self._hyper_dev = _to_device(NativeCompressor._default_hyper(), device)
        self._key = key
        self._tapes.clear()
        self._choose_path(total, world_size(), device)

    def _choose_path(self, total: int, workers: int, device: torch.device) -> None:
        """local | oneshot (flag-in-data words to every peer) | bulk (two-shot, plain floats +
        chunk flags; the flat buffer lives in the symmetric arena; PSGD_B200_FLAT=bulk forces it
        for small buffers too) | nvls (PSGD_B200_FLAT=nvls: in-switch reduction of a buffer bound to
        an NVLink multicast object, for buffers above the one-shot limit) | nccl
        (PSGD_B200_COMM=nccl, or arena too large)."""
        want = os.environ.get("PSGD_B200_FLAT", "auto")
        p2p = workers > 1 and os.environ.get("PSGD_B200_COMM", "p2p") == "p2p"
        self.n_pad = total
        if workers == 1:
            path, cap = "local", 0
        elif not p2p:
            path, cap = "nccl", 0
        elif total <= self.ONE_SHOT_LIMIT_FLOATS and want != "bulk":
            path, cap = "oneshot", total
        elif self._wants_nvls(want, workers) and self._nvls_buffer(total) is not None:
            path, cap = "nvls", 0
            self.n_pad = self._nvls.n_pad
        else:
            unit = workers * int(self.lib.psgd_bulk_chunk_floats())
            self.n_pad = -(-total // unit) * unit
            nbytes = int(self.lib.psgd_bulk_arena_bytes(ctypes.c_longlong(self.n_pad), workers))
            path, cap = "bulk", -(-nbytes // (16 * workers))
        if cap and 2 * workers * cap * 8 > self.P2P_ARENA_LIMIT_BYTES:
            path, cap = "nccl", 0
        # An arena is reused only under the discipline it was written with: flag-in-data words of
        # old epochs never match a new one, but the bulk layout puts its flag tables where another
        # layout had data, so a change of protocol or of the bulk size starts from a zeroed arena.
        bulk_layout = self.n_pad if path == "bulk" else None
        if self.comm is not None and (self.comm.cap < cap or cap == 0 or bulk_layout != self._bulk_layout):
            self.comm.close()
            self.comm = None
        self._bulk_layout = bulk_layout
        if cap and self.comm is None:
            from .parallel.symm import Channel

            self.comm = Channel(cap)
        if path in ("nccl", "oneshot"):
            self._flat = torch.zeros(total, device=device, dtype=torch.float32)
        elif path == "local":
            self._flat = None   # one worker: nothing is packed
        elif path == "bulk":
            # pack writes and unpack reads the arena's data region directly
            self._flat = self.comm.slots.tensor(0, self.n_pad)
        elif path == "nvls":
            self._flat = self._nvls.buffer  # this rank's replica of the multicast-bound buffer
        if path != "nvls" and self._nvls is not None:
            self._nvls.close()
            self._nvls = None
        self.path = path

    @staticmethod
    def _wants_nvls(want: str, workers: int) -> bool:
        """In-switch reduction for buffers above the one-shot limit: always with
        PSGD_B200_FLAT=nvls; by default from four workers on (measured at four GPUs: 10-27 % faster
        than the library all-reduce from 1 MiB to 268 MB, where the two-shot peer-store kernels are
        12-35 % behind it; at two GPUs the peer-store kernels are as fast as either). Setting
        NCCL_NVLS_ENABLE=0 - the switch that keeps the communication library off NVLink multicast -
        keeps this path off too, which is how the failure tests run."""
        if want == "nvls":
            return True
        return want == "auto" and workers >= 4 and os.environ.get("NCCL_NVLS_ENABLE", "1") != "0"

    def _nvls_buffer(self, total: int):
        """The in-switch all-reduce object for `total` floats, or None when the machine offers no
        NVLink multicast (every rank decides alike; a warning is printed once)."""
        if self._nvls is not None and self._nvls.n_pad >= total:
            return self._nvls
        if self._nvls_failed:
            return None
        from .parallel.nvls import NvlsAllReduce, NvlsUnavailable

        if self._nvls is not None:
            self._nvls.close()
            self._nvls = None
        try:
            self._nvls = NvlsAllReduce(total)
        except NvlsUnavailable as exc:
            import warnings

            warnings.warn(f"in-switch all-reduce not available ({exc}); using the peer-store kernels")
            self._nvls, self._nvls_failed = None, True
        return self._nvls

    def _launch(self, mode: int, hyper_dev: torch.Tensor, divisor: float, early: bool = False,
                stream: Optional[ctypes.c_void_p] = None) -> None:
        code = self.lib.psgd_flat_launch(
            mode,
            self._vec,
            _ptr(self._items_dev),
            _ptr(self._block_item),
            _ptr(self._block_first),
            self._nblocks,
            _ptr(hyper_dev),
            _ptr(self._flat),
            float(divisor),
            self.comm.ptr if self.comm is not None else ctypes.c_void_p(0),
            ctypes.c_longlong(self.n_pad),
            1 if self._keep_inputs else 0,
            int(early),
            _stream_ptr() if stream is None else stream,
        )
        native.check(code, "psgd_flat_launch")
        self.launches += 1

    def _owned(self) -> tuple:
        return self._items_dev, self._block_item, self._block_first, self._hyper_dev, self._flat, self._out

    def _run(self, hyper_dev: torch.Tensor, workers: int, sgd: bool, early: bool = False, inside: bool = False) -> None:
        stream = _stream_ptr()
        if stream and not inside and is_recorded(stream):   # (0, the default stream: never)
            with self._being_recorded(stream):
                keep_with_graph(self._kept, hyper_dev)
                self._run(hyper_dev, workers, sgd, early, inside=True)
            return
        self._stream = stream
        if self.path == "local":
            key = (sgd, early, self._keep_inputs, hyper_dev.data_ptr())
            tape = self._tapes.get(key)
            if tape is not None:
                tape(stream)
                self.launches += tape.count
                return
            before = self.launches
            tape = _Tape(self.lib, lambda: self._launch(4 if sgd else 3, hyper_dev, 1.0, early, stream=stream))
            if tape.count == self.launches - before:   # (it went through the library's one way of launching)
                if len(self._tapes) >= 16:
                    self._tapes.clear()
                self._tapes[key] = tape
        elif self.path == "bulk":
            self._launch(0, hyper_dev, float(workers), stream=stream)
            code = self.lib.psgd_bulk_allreduce_launch(self.comm.ptr, ctypes.c_longlong(self.n_pad), workers, _stream_ptr())
            native.check(code, "psgd_bulk_allreduce_launch")
            self.launches += 2
            self._launch(13 if sgd else 12, hyper_dev, 1.0, stream=stream)
        elif self.path == "nvls":
            self._launch(0, hyper_dev, float(workers), stream=stream)
            self._nvls.all_reduce_()
            self.launches += self._nvls.launches
            self._launch(2 if sgd else 1, hyper_dev, 1.0, stream=stream)
        elif self.path == "oneshot":
            if self._pushed:
                self._pushed = False
            else:
                self._launch(5, hyper_dev, float(workers), stream=stream)
            self._launch(7 if sgd else 6, hyper_dev, 1.0, stream=stream)
        else:
            self._launch(0, hyper_dev, float(workers), stream=stream)
            dist.all_reduce(self._flat)
            self._launch(2 if sgd else 1, hyper_dev, 1.0, stream=stream)

    def aggregate(self, gradients: List[torch.Tensor], outs: Optional[Sequence[torch.Tensor]] = None,
                  keep_inputs: bool = False, early: bool = False) -> List[torch.Tensor]:
        """Mean over workers. `outs`: caller-owned destination tensors (default: views of this
        object's buffer, valid until the next call). `keep_inputs`: do not zero the inputs. `early`: see `aggregate_and_step`."""
        self.check()
        self.launches = 0
        self._bind(gradients, outs=outs)
        self._keep_inputs = bool(keep_inputs)
        try:
            self._run(self._hyper_dev, world_size(), sgd=False, early=early)
        finally:
            self._keep_inputs = False
        return list(self._views)

    def aggregate_and_step(self, gradients, params, moms, hyper_index, hyper_dev, early: bool = False) -> None:
        """The mean and the optimizer step in one pass. `early`: the launch before this one is the
        decompression of other tensors, whose end it may overlap (one worker)."""
        self.check()
        self.launches = 0
        self._bind(gradients, params, moms, hyper_index, need_out=False)
        self._run(hyper_dev, world_size(), sgd=True, early=early)

    def close(self) -> None:
        """Release the symmetric arena (collective across ranks)."""
        if self.comm is not None:
            self.comm.close()
            self.comm = None
        if self._nvls is not None:
            self._nvls.close()
            self._nvls = None
        self._key = None
        self._bulk_layout = None


class MultiTensorAccumulate:
    """`dst[i] += src[i]` for two lists of float32 tensors in ONE launch.

    Error feedback keeps the compression residual in `p.grad` and lets autograd accumulate the
    next gradient onto it (powersgd/__init__.py:17-25), which costs one small add kernel per
    parameter. A training step that owns the loop detaches the residuals before backward, lets
    autograd adopt the fresh gradients without arithmetic, and folds them in with this kernel.

    Multi-GPU: the same launch can carry the first half of the flat all-reduce of the uncompressed
    tensors (`push=`): their gradients are scaled, zeroed and pushed into every peer's slots while
    the residuals are folded, so that the data is on its way before the low-rank kernels start."""

    def __init__(self):
        self.lib = native.lib()
        self._key = None
        self._kept: dict = {}   # tables that recorded launches refer to

    def __call__(self, dst: Sequence[torch.Tensor], src: Sequence[torch.Tensor], push: "Optional[NativeFlatAllReduce]" = None) -> None:
        key = (tuple(t.data_ptr() for t in dst), tuple(t.data_ptr() for t in src), None if push is None else push._key)
        if key != self._key:
            device = dst[0].device
            per_block = self.lib.psgd_flat_block_elems()
            pushed = [] if push is None else list(np.frombuffer(push._items_host.tobytes(), dtype=layout.FLAT_DTYPE))
            items = np.zeros(len(dst) + len(pushed), dtype=layout.FLAT_DTYPE)
            block_item, block_first = [], []
            for i, (d, s_) in enumerate(zip(dst, src)):
                if not same_layout(d, s_) or d.dtype != torch.float32 or s_.dtype != torch.float32:
                    raise ValueError("accumulate needs float32 tensors of equal shape and layout")
                if not is_dense(d):
                    raise ValueError("accumulate needs dense tensors")
                items[i]["grad"], items[i]["out"], items[i]["numel"] = s_.data_ptr(), d.data_ptr(), d.numel()
                items[i]["op"] = 8
            for j, it in enumerate(pushed):
                items[len(dst) + j] = it
                items[len(dst) + j]["op"] = 5
            for i in range(len(items)):
                for first in range(0, int(items[i]["numel"]), per_block):
                    block_item.append(i)
                    block_first.append(first)
            self._vec = 1 if all(ptr % 16 == 0 for ptr in key[0] + key[1]) else 0
            self._items = _to_device(items, device)
            self._block_item = _to_device(np.asarray(block_item, dtype=np.int32), device)
            self._block_first = _to_device(np.asarray(block_first, dtype=np.int32), device)
            self._nblocks = len(block_item)
            self._hyper = _to_device(NativeCompressor._default_hyper(), device)
            self._key = key
        stream = _stream_ptr()
        if is_recorded(stream):
            keep_with_graph(self._kept, self._items, self._block_item, self._block_first, self._hyper)
        code = self.lib.psgd_flat_launch(
            8 if push is None else 9, self._vec, _ptr(self._items), _ptr(self._block_item), _ptr(self._block_first),
            self._nblocks, _ptr(self._hyper), ctypes.c_void_p(0), 1.0 if push is None else float(world_size()),
            ctypes.c_void_p(0) if push is None else push.comm.ptr, ctypes.c_longlong(0), 0, 0, stream,
        )
        native.check(code, "psgd_flat_launch")
        if push is not None:
            push._pushed = True


class FusedSGDDriver:
    """Glue between `torch.optim.SGD` and the fused kernels.

    Keeps `optimizer.state[p]["momentum_buffer"]` as the live momentum tensors (so optimizer
    checkpoints stay valid), refreshes a small device table of per-group hyper-parameters
    every step (learning-rate schedules keep working), and follows torch's first-step rule
    that a fresh momentum buffer is the gradient itself.

    The table travels through a ring of pinned host slots, one async copy per step that changes
    it, so that a step recorded in a CUDA graph reads its hyper-parameters from device memory and
    the host never overwrites a slot that a copy in flight still reads. No copy is ever recorded:
    a recorded step runs with what the device table holds when it is replayed (`prepare`, or any
    eager step, brings it up to date).
    """

    RING = 4

    def __init__(self, agg):
        self.agg = weakref.proxy(agg)   # its owner, see NativeCompressor
        self.lib = native.lib()
        self.device = agg.device
        self._slots: List[torch.Tensor] = []
        self._slot_events: List[Optional[torch.cuda.Event]] = []
        self._cursor = 0
        self._hyper_dev: Optional[torch.Tensor] = None
        self._cache_key = None
        self._last_values = None   # what the device table holds
        self._fixed: Optional[torch.Tensor] = None   # table of the coming step alone, in place of the live one
        self._flat_all = NativeFlatAllReduce()
        self._flat_plain = NativeFlatAllReduce()
        self.launches = 0

    def _collect(self, optimizer):
        groups = optimizer.param_groups
        key = (id(optimizer), tuple(len(g["params"]) for g in groups), tuple(float(g["momentum"]) != 0.0 for g in groups))
        fresh_groups = set()
        # a group whose first buffer is missing or another tensor (a loaded optimizer checkpoint) is looked at anew
        if key != self._cache_key or any(
            float(g["momentum"]) != 0.0 and optimizer.state[p].get("momentum_buffer") is not first
            for g, first in zip(groups, self._first_moms)
            for p in g["params"][:1]
        ):
            params, moms, index = [], [], []
            for gi, group in enumerate(groups):
                mu = float(group["momentum"])
                for p in group["params"]:
                    params.append(p)
                    index.append(gi)
                    if mu != 0.0:
                        st = optimizer.state[p]
                        if st.get("momentum_buffer") is None:
                            st["momentum_buffer"] = torch.zeros_like(p)  # preserve_format: laid out like the parameter
                            fresh_groups.add(gi)
                        moms.append(st["momentum_buffer"])
                    else:
                        moms.append(None)
            self._params, self._moms, self._index = params, moms, index
            self._first_moms = [optimizer.state.get(g["params"][0], {}).get("momentum_buffer") if g["params"] else None for g in groups]
            mask = self.agg.is_compressed_mask
            if len(params) == len(mask):
                # the same lists, compressed and uncompressed tensors apart (True / False)
                self._split = {keep: tuple([x for x, k in zip(xs, mask) if k == keep] for xs in (params, moms, index))
                               for keep in (True, False)}
            self._bound_grads = None
            self._cache_key = key
        return fresh_groups

    def prepare(self, optimizer) -> None:
        """Host side of a step: momentum buffers, hyper-parameter table, async upload."""
        fresh = self._collect(optimizer)
        groups = optimizer.param_groups
        # one row per group, as the kernels see it: a fresh momentum buffer is the gradient itself, whatever the dampening
        values = [
            (float(g["lr"]), float(g["momentum"]), 1.0 if gi in fresh else 1.0 - float(g["dampening"]), float(g["weight_decay"]), bool(g["nesterov"]))
            for gi, g in enumerate(groups)
        ]
        self._fixed = None
        if values == self._last_values:
            return  # nothing changed since the last upload: the device table is already right
        table = np.zeros(len(groups), dtype=layout.HYPER_DTYPE)
        for row, (lr, mu, one_minus_dampening, decay, nesterov) in zip(table, values):
            row["lr"] = lr
            row["momentum"] = mu
            row["one_minus_dampening"] = one_minus_dampening
            row["weight_decay"] = decay
            row["nesterov"] = 1 if nesterov else 0
            row["has_momentum"] = 1 if mu != 0.0 else 0
            row["grad_scale"] = 1.0
        stream = _stream_ptr()
        recording = native.capture_id(stream) if is_recorded(stream) else 0
        readers = [r for r in (self.agg._powersgd._native, self._flat_all, self._flat_plain) if r is not None]
        streams = [r._stream for r in readers if r._stream is not None]
        if recording and (any(r.recorded_in == recording for r in readers) or any(s and native.capture_id(s) for s in streams)):
            # The live table cannot change under a step that reads it already: one recorded before this in the
            # same graph, or one that may still be running on a stream that is part of the recording and so
            # cannot be waited for. This step keeps the values it was recorded with.
            self._fixed = _to_device(table, self.device)
            return
        nbytes = table.nbytes
        if self._hyper_dev is None or self._hyper_dev.numel() != nbytes:
            with outside_capture(self.device):
                self._slots = [torch.empty(nbytes, dtype=torch.uint8).pin_memory() for _ in range(self.RING)]
                self._slot_events = [None] * self.RING
                self._hyper_dev = torch.empty(nbytes, dtype=torch.uint8, device=self.device)
        self._last_values = values
        raw = table.view(np.uint8).reshape(-1)
        if recording:
            # in place now, not by a copy that every replay would repeat over what later steps upload
            with outside_capture(self.device):
                for stream in streams:   # the steps before this one have read the table
                    native.check(self.lib.psgd_stream_wait(stream), "psgd_stream_wait")
                self._hyper_dev.copy_(torch.from_numpy(raw))
            return
        i = self._cursor
        self._cursor = (i + 1) % self.RING
        if self._slot_events[i] is not None:
            self._slot_events[i].synchronize()
        self._slots[i].numpy()[:] = raw
        self._hyper_dev.copy_(self._slots[i], non_blocking=True)
        ev = torch.cuda.Event()
        ev.record()
        self._slot_events[i] = ev

    def check(self) -> None:
        """Raise `PowerSGDCommTimeout` if any bounded device-side wait of an earlier step gave up:
        a peer that stayed away leaves zeros in place of its contribution, so the step that
        follows must not run. Host reads of mapped pinned words only; called every step."""
        core = self.agg._powersgd
        if core._native is not None:
            core._native.check()
        self._flat_all.check()
        self._flat_plain.check()

    def fold(self, accumulate: "MultiTensorAccumulate", dst: Sequence[torch.Tensor], src: Sequence[torch.Tensor]) -> None:
        """`dst[i] += src[i]` (residual + fresh gradient) in one launch which, on several GPUs in
        the compression phase, also packs and pushes the uncompressed tensors' gradients."""
        agg = self.agg
        push = None
        if world_size() > 1 and agg.step_counter >= agg.config.start_compressing_after_num_steps and getattr(self, "_params", None):
            mask = agg.is_compressed_mask
            pick = lambda xs: [x for x, k in zip(xs, mask) if not k]  # noqa: E731
            plain = [p.grad for p in pick(self._params)]
            if plain and all(g is not None for g in plain):
                flat = self._flat_plain
                flat._bind([g.data for g in plain], pick(self._params), pick(self._moms), pick(self._index), need_out=False)
                if flat.path == "oneshot":
                    push = flat
        accumulate(dst, src, push=push)

    def step(self, optimizer, prepared: bool = False) -> None:
        self.check()
        if not prepared:
            self.prepare(optimizer)
        # the gradient tensors may have been replaced since the last step (dropped zero gradients
        # re-created by autograd, a loaded checkpoint): always bind what the parameters hold now
        agg = self.agg
        mask = agg.is_compressed_mask
        now = scan.grad_addresses(self._params)
        if now != self._bound_grads:
            self._grads = [p.grad.data for p in self._params]
            self._split_grads = {keep: [g for g, k in zip(self._grads, mask) if k == keep] for keep in (True, False)}
            self._bound_grads = now
        hyper_dev = self._hyper_dev if self._fixed is None else self._fixed
        self._fixed = None
        index, params, moms, grads = self._index, self._params, self._moms, self._grads
        if len(grads) != len(mask):
            raise ValueError("optimizer parameters do not match the aggregator's parameter list")
        agg.step_counter += 1
        if agg.step_counter <= agg.config.start_compressing_after_num_steps:
            self._flat_all.aggregate_and_step(grads, params, moms, index, hyper_dev)
            self.launches = self._flat_all.launches
            return
        core = agg._powersgd
        self.launches = 0
        if core.params:
            if core._native is None:
                core._native = NativeCompressor(core)
            core._native.aggregate_and_step(self._split_grads[True], *self._split[True], hyper_dev)
            core.step_counter += 1
            self.launches += core._native.launches
        plain = self._split_grads[False]
        if plain:
            # after the low-rank path: a consumer that spins on its peers next to the product
            # kernels (tried as a parallel side-stream branch) cost more than it hid
            self._flat_plain.aggregate_and_step(
                plain, *self._split[False], hyper_dev,
                early=bool(core.params) and core._native._chained(),
            )
            self.launches += self._flat_plain.launches
