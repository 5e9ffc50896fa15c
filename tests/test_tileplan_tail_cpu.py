"""Tensor-core tiles of lists of more than one round of resident CTAs, whose last output blocks are cut finer (host code only)."""
import pytest

from powersgd_b200.plan import CompressionPlan

native = pytest.importorskip("powersgd_b200.ops.native")


@pytest.mark.parametrize("shapes,rank", [([(50257, 1024)], 16), ([(38016, 256)], 9), ([(37889, 1000)], 11), ([(20000, 640)] * 4, 8),
                                         ([(4096, 4096)] * 4, 4), ([(512, 38000)], 32), ([(24000, 1500), (130, 40004), (9000, 132)], 11)])
def test_every_sum_is_covered_once_and_the_last_round_is_full(shapes, rank):
    from powersgd_b200.cuda_path import TilePlan

    plan = CompressionPlan.build(shapes, rank=rank)
    try:
        tiles = TilePlan(plan, native.lib())
    except Exception as exc:
        pytest.skip(f"native library unavailable: {exc}")
    tiles.fin_rows = 256
    arrays = tiles.build([4] * len(tiles.mats), [True] * len(tiles.mats))
    slots = 148 * TilePlan.TC_CTAS_PER_SM
    for name, along, size in (("nt", "row0", "rows"), ("nn", "col0", "cols")):
        by_ticket = {}
        for t in arrays[name]["tc"]:
            by_ticket.setdefault(int(t["ticket"]), []).append(t)
        for group in by_ticket.values():
            at = 0
            for i, t in enumerate(group):
                assert (int(t["split"]), int(t["nsplit"])) == (i, len(group)) and int(t[along]) == at and at % 32 == 0
                at += int(t[size])
            g = plan.groups[tiles.mats[int(group[0]["mat"])][0]]
            assert at == (g.n if name == "nt" else g.m)
        count = len(arrays[name]["tc"])
        blocks = sum(g.batch * -(-(g.m if name == "nt" else g.n) // 128) for g in plan.groups)
        assert len(by_ticket) == blocks
        if rank > 8 and slots < blocks <= 1.5 * slots:   # the rest of the blocks has room to be cut at least in two
            last = arrays[name]["tc"][-1]
            g = plan.groups[tiles.mats[int(last["mat"])][0]]
            assert count > blocks and int(last[size]) <= (g.n if name == "nt" else g.m) / 2 + 32
