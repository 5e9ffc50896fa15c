"""Segments of the one-pass kernel for the last product and the decompression (host code; needs the built library)."""
import os

import numpy as np
import pytest

from powersgd_b200.plan import CompressionPlan

native = pytest.importorskip("powersgd_b200.ops.native")


@pytest.mark.parametrize("rank,iters", [(1, 1), (1, 4), (2, 2), (3, 2), (4, 2), (8, 1)])
def test_segments_cover_every_row_once_and_fit_the_kernel(rank, iters):
    from powersgd_b200.cuda_path import TilePlan

    try:
        lib = native.lib()
    except Exception as exc:
        pytest.skip(f"native library unavailable: {exc}")
    shapes = [(64, 27), (10, 512), (1000, 650), (512, 4608), (5, 9), (4096, 1024), (24000, 24), (333, 129), (3, 1001)]
    tiles = TilePlan(CompressionPlan.build(shapes, rank=rank), lib)
    of = lambda mi: tiles.plan.groups[tiles.mats[mi][0]]  # noqa: E731
    rows_of = lambda m, n: int(lib.psgd_panel_rows(tiles.max_r, iters, m, n))  # noqa: E731
    mats = [mi for mi in range(len(tiles.mats)) if rows_of(of(mi).m, of(mi).n)]
    assert len(mats) >= 8
    segs, starts = tiles.panel_segments(mats, [1] * len(tiles.mats), rows_of)
    assert starts[0] == 0 and starts[-1] == len(segs) and (np.diff(starts) >= 0).all() and len(starts) <= 149
    seen = {mi: np.zeros(of(mi).n, dtype=int) for mi in mats}
    for s in segs:
        g = of(s["mat"])
        assert s["row0"] % 4 == 0 and (s["rows"] % 4 == 0 or s["row0"] + s["rows"] == g.n) and s["cols"] == g.m
        assert s["split"] > 0 and s["split"] % 4 == 0
        seen[int(s["mat"])][s["row0"] : s["row0"] + s["rows"]] += 1
    assert all((rows == 1).all() for rows in seen.values())
    work = [sum(int(s["rows"]) * int(s["cols"]) for s in segs[a:b]) for a, b in zip(starts, starts[1:])]
    total = sum(of(mi).n * of(mi).m for mi in mats)
    assert max(work) <= total / len(work) + 8 * 4608   # a quad of the widest matrix at either end


def _plan(shapes, rank, iters):
    """(the plan, matrices that the kernel takes, factor columns, rows per panel)"""
    from powersgd_b200.cuda_path import TilePlan

    try:
        lib = native.lib()
    except Exception as exc:
        pytest.skip(f"native library unavailable: {exc}")
    tiles = TilePlan(CompressionPlan.build(shapes, rank=rank), lib)
    rows_of = lambda m, n: int(lib.psgd_panel_rows(tiles.max_r, iters, m, n))  # noqa: E731
    size = [(tiles.plan.groups[gi].n, tiles.plan.groups[gi].m) for gi, _pos, _idx in tiles.mats]
    return tiles, size, [mi for mi, (n, m) in enumerate(size) if rows_of(m, n)], tiles.rt * iters, rows_of


def _widths(size):
    return [4 if m % 4 == 0 else 2 if m % 2 == 0 else 1 for _n, m in size]


MANY_SMALL = [(1024, 1024)] * 8 + [(64, 64)] * 20


@pytest.mark.parametrize("rank,iters", [(1, 2), (2, 2), (4, 2), (8, 1)])
@pytest.mark.parametrize("shapes", [MANY_SMALL, [(1024, 1024)] * 8 + [(8000, 24)], [(2048, 2048)] * 4 + [(1000, 131)] * 4, [(512, 1024)] * 3])
def test_no_block_gets_most_of_the_small_segments(shapes, rank, iters):
    """Starts and narrow rows count: the blocks' costs are alike up to a quad and a start at either end."""
    tiles, size, mats, columns, rows_of = _plan(shapes, rank, iters)
    row, start = tiles.panel_costs(mats, _widths(size), columns)
    segs, starts = tiles.panel_segments(mats, _widths(size), rows_of, row, start)
    rows = np.zeros(len(size), dtype=np.int64)
    np.add.at(rows, segs["mat"], segs["rows"])
    assert rows.tolist() == [n for n, _m in size] and starts[0] == 0 and starts[-1] == len(segs)
    least = dict(zip(mats, row.tolist()))
    cost = [sum(start + int(s["rows"]) * max(int(s["cols"]), least[int(s["mat"])]) for s in segs[a:b]) for a, b in zip(starts, starts[1:])]
    widest = max(max(m, r) for (_n, m), r in zip(size, row))
    total = sum(start + n * max(m, least[mi]) for mi, (n, m) in enumerate(size))
    assert max(cost) <= total / len(cost) + 2 * start + 8 * widest


@pytest.mark.parametrize("shapes,rank,iters,pays", [
    ([(4096, 4096)] * 4, 4, 2, True),
    (MANY_SMALL, 4, 2, True),
    ([(1024, 1024)] * 8 + [(64, 64)] * 300, 2, 2, False),     # starts
    ([(64, 64)] * 500, 1, 2, False),
    ([(24000, 96)] * 4, 1, 2, False),                         # narrow rows
    ([(512, 2304)] * 2 + [(1000, 131)] * 4, 1, 2, False),
    ([(4, 4096)] * 100, 4, 2, True),                          # few rows
    ([(700, 1024)] * 2, 1, 2, False),                         # too little
    ([(780, 1024)] * 2, 1, 2, True),
    ([(780, 1024)] * 2, 4, 2, False),                         # ... for eight factor columns
    ([(2048, 2048)] * 2, 8, 1, False),                        # ... for a product of rank 8 on the tensor cores
    ([(2048, 2048)] * 4, 8, 1, True),
    ([(512, 4608)] * 3 + [(512, 2304)] * 8, 4, 2, False),     # some are too wide for the kernel
    ([(512, 4608)] * 3 + [(512, 2304)] * 8, 2, 2, True),
])
def test_where_one_pass_pays(shapes, rank, iters, pays):
    from powersgd_b200.cuda_path import NativeCompressor

    tiles, size, mats, columns, _rows_of = _plan(shapes, rank, iters)
    tc = [m % 4 == 0 and n >= 128 and m >= 128 and (rank >= 8 or sum(a * b for a, b in size) > 24 << 20) for n, m in size]
    assert tiles.panel_pays(mats, _widths(size), columns, tc, NativeCompressor.PANEL_ELEMS) == pays


def test_refused_shapes():
    try:
        lib = native.lib()
    except Exception as exc:
        pytest.skip(f"native library unavailable: {exc}")
    for rank, iters, m in [(9, 1, 64), (8, 2, 64), (4, 3, 64), (1, 5, 64), (4, 2, 4097), (8, 1, 4097), (1, 1, 7000)]:
        assert lib.psgd_panel_rows(rank, iters, m, 1000) == 0
    for rank, iters, m in [(4, 2, 4096), (2, 2, 4608), (8, 1, 4096)]:
        assert lib.psgd_panel_rows(rank, iters, m, 1000) == 4


def test_stores_of_a_segment_are_fenced_from_the_copies_of_the_next():
    """Where the rings begin depends on the height of a panel, so the copies of one segment may land on bytes that the
    one before stored (tests/test_panel_gpu.py, test_segments_of_unlike_matrices): every thread has to fence."""
    with open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "powersgd_b200", "csrc", "panel.cu")) as fp:
        loop = fp.read().split("for (int s = first; s < end; ++s) {")[1]
    assert 0 < loop.find("psgd_fence_async_shared();") < loop.find("__syncthreads();") < loop.find("sg.tile = a.tiles[s];")
