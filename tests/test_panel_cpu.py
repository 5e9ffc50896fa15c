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
