"""The grouped products against float64 at the edges of their tiles."""
import pytest
import torch

from powersgd_b200 import BasicConfig, BasicPowerSGD

pytestmark = pytest.mark.gpu

# row and column counts around a warp's rows, a tile's rows and columns and a staged stretch of
# columns; pitches that allow 16-, 8- and 4-byte accesses
SHAPES = [(31, 127), (32, 128), (33, 129), (40, 27), (128, 510), (129, 1023), (95, 1024), (97, 1025), (257, 1154), (70, 2052), (5000, 66)]


@pytest.mark.parametrize("rank", [1, 2, 3, 4, 8, 11, 16, 27])
def test_products_at_tile_edges(rank, monkeypatch):
    """A running sum of products in float32 with independent roundings is off by about 0.7 * 2^-24 of
    |row| |column|; four times 2^-24, over the whole product."""
    monkeypatch.setenv("PSGD_B200_GEMM", "ffma")
    core = BasicPowerSGD([torch.zeros(s, device="cuda") for s in SHAPES], BasicConfig(rank=rank, num_iters_per_step=1), backend="native")
    g = torch.Generator(device="cuda").manual_seed(rank)
    grads = [torch.randn(s, generator=g, device="cuda") for s in SHAPES]
    keep = [x.clone() for x in grads]
    core.aggregate(grads)
    nat = core._native
    for x, k in zip(grads, keep):
        x.copy_(k)   # the tensors the compressor is bound to
    for transposed in (True, False):
        fac, out = nat.h_in[0], nat.h_loc[0]
        fac.copy_(torch.randn(fac.shape, generator=g, device="cuda"))
        out.fill_(float("nan"))
        nat._gemm(transposed, fac, out, [], [])
        for grp in core.plan.groups:
            offs = (grp.p_offset, grp.q_offset, grp.n, grp.m)
            (i0, o0, ni, no) = offs if transposed else (offs[1], offs[0], offs[3], offs[2])
            for pos, idx in enumerate(grp.members):
                f = fac[i0 + pos * ni * grp.r : i0 + (pos + 1) * ni * grp.r].view(ni, grp.r).double()
                got = out[o0 + pos * no * grp.r : o0 + (pos + 1) * no * grp.r].view(no, grp.r).double()
                m = keep[idx].double()
                want = (m.T if transposed else m) @ f
                bound = 4 * 2.0 ** -24 * m.norm() * f.norm()
                assert (got - want).norm() <= bound, (SHAPES[idx], transposed)
