"""Tensor-core tiles of lists of more than one round of resident CTAs, whose last output blocks are cut finer (host code only)."""
import heapq

import pytest

from powersgd_b200.plan import CompressionPlan

native = pytest.importorskip("powersgd_b200.ops.native")
MIXED = [([(24000, 1500), (130, 40004), (9000, 132)], 11), ([(2072, 7932), (4760, 5784), (1808, 5220), (35986, 568)], 11),
         ([(20336, 672)] * 3 + [(464, 3952), (5328, 480), (1856, 2864)], 11), ([(28000, 130)] * 2 + [(700, 30000)], 16), ([(25718, 460)] * 2, 16)]


def _plan(shapes, rank):
    from powersgd_b200.cuda_path import TilePlan

    try:
        lib = native.lib()
    except Exception as exc:
        pytest.skip(f"native library unavailable: {exc}")
    tiles = TilePlan(CompressionPlan.build(shapes, rank=rank), lib)
    tiles.fin_rows = 256
    return tiles


def _end(lengths, overhead, slots):
    """When the last CTA ends if the tiles go to the first place that is free, one after another."""
    ends = [0] * slots
    for n in lengths:
        heapq.heapreplace(ends, ends[0] + overhead + int(n))
    return max(ends)


@pytest.mark.parametrize("shapes,rank", [([(50257, 1024)], 16), ([(38016, 256)], 9), ([(37889, 1000)], 11), ([(20000, 640)] * 4, 8),
                                         ([(4096, 4096)] * 4, 4), ([(512, 38000)], 32)] + MIXED)
def test_every_sum_is_covered_once_and_the_last_round_ends_no_later(shapes, rank, monkeypatch):
    tiles = _plan(shapes, rank)
    plan = tiles.plan
    arrays = tiles.build([4] * len(tiles.mats), [True] * len(tiles.mats))
    slots, overhead = 148 * tiles.TC_CTAS_PER_SM, tiles.TC_ROUND_OVERHEAD_ROWS
    monkeypatch.setattr(tiles, "_tc_extents", lambda groups, transposed: (tiles._pick_tc_k(groups, transposed), {}))
    plain = tiles.build([4] * len(tiles.mats), [True] * len(tiles.mats))
    for name, along, size in (("nt", "row0", "rows"), ("nn", "col0", "cols")):
        by_ticket = {}
        for t in arrays[name]["tc"]:
            by_ticket.setdefault(int(t["ticket"]), []).append(t)
        for group in by_ticket.values():
            at = 0
            for i, t in enumerate(group):
                assert (int(t["split"]), int(t["nsplit"])) == (i, len(group)) and int(t[along]) == at and at % 32 == 0
                assert int(t[size]) <= tiles.TC_MAX_EXTENT
                at += int(t[size])
            g = plan.groups[tiles.mats[int(group[0]["mat"])][0]]
            assert at == (g.n if name == "nt" else g.m)
        count = len(arrays[name]["tc"])
        blocks = sum(g.batch * -(-(g.m if name == "nt" else g.n) // 128) for g in plan.groups)
        assert len(by_ticket) == blocks
        last = arrays[name]["tc"][-1]
        g = plan.groups[tiles.mats[int(last["mat"])][0]]
        length = g.n if name == "nt" else g.m
        # the rest of the blocks has room to be cut at least in two (halves of a sum shorter than this save less than a tenth)
        if len(plan.groups) == 1 and rank > 8 and slots < blocks <= 1.5 * slots and length / 2 + overhead < 0.8 * (length + overhead):
            assert count > blocks and int(last[size]) <= length / 2 + 32
        for mi in range(len(tiles.mats)):   # no worse sums: chains of at most 512 terms in the tensor core, off by the 3/2th power of their length each
            off = lambda lists: {t: sum(int(x) // 512 * 512 ** 3 + (int(x) % 512) ** 3 for x in lists[size][lists["ticket"] == t])  # noqa: E731
                                 for t in set(lists["ticket"][lists["mat"] == mi].tolist())}
            assert max(off(arrays[name]["tc"]).values()) <= max(off(plain[name]["tc"]).values())
        ends, before = _end(arrays[name]["tc"][size], overhead, slots), _end(plain[name]["tc"][size], overhead, slots)
        assert ends <= before
        if rank <= 8 or not slots < len(plain[name]["tc"]) <= 3 * slots:
            assert count == len(plain[name]["tc"])


def test_the_finest_cut_that_the_example_gives():
    """50257 x 1024 at rank 16, M Q: 296 blocks in one tile each, the 97 behind them in three, so that both rounds are full."""
    tiles = _plan([(50257, 1024)], 16)
    cols = tiles.build([4], [True])["nn"]["tc"]["cols"].tolist()
    assert cols[:296] == [1024] * 296 and len(cols) == 296 + 3 * 97 and max(cols[296:]) <= 352
