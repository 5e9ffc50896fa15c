"""Launches made again from the library's own record: as many as the step reported, dropped with the binding, recorded anew for
another learning-rate table, and of the same bits on another stream."""
import pytest
import torch

from powersgd_b200 import Config, PowerSGD, optimizer_step

pytestmark = pytest.mark.gpu

SHAPES = [(300, 200), (64, 3, 3, 3), (77,), (1001, 130)]


@pytest.mark.parametrize("momentum", [0.0, 0.9])
@pytest.mark.parametrize("warmup", [0, 1000])
def test_repeated_steps(momentum, warmup):
    def run(forget):
        g = torch.Generator(device="cuda").manual_seed(2)
        draw = lambda: [torch.randn(s, generator=g, device="cuda") for s in SHAPES]  # noqa: E731
        params = [torch.nn.Parameter(p) for p in draw()]
        agg = PowerSGD(params, Config(rank=3, num_iters_per_step=3, start_compressing_after_num_steps=warmup))
        opt = torch.optim.SGD(params, lr=0.1, momentum=momentum)
        side = torch.cuda.Stream()
        for step in range(9):
            fresh = draw()
            if step in (0, 6):   # other tensors from here on
                for p, f in zip(params, fresh):
                    p.grad = f.clone()
            else:
                torch._foreach_add_([p.grad for p in params], fresh)
            nat = agg._powersgd._native
            driver = getattr(agg, "_fused", None)
            if forget and driver is not None:
                for holder in (nat, driver._flat_all, driver._flat_plain):
                    if holder is not None:
                        holder._tapes.clear()
            opt.param_groups[0]["lr"] = 0.1 / (1 + step // 4)
            torch.cuda.synchronize()
            with torch.cuda.stream(side if step == 4 else torch.cuda.current_stream()):
                optimizer_step(opt, agg)
            torch.cuda.synchronize()
        return [p.detach().clone() for p in params] + [p.grad.clone() for p in params], agg

    (usual, agg), (anew, _) = run(False), run(True)
    assert all(torch.equal(a, b) for a, b in zip(usual, anew))
    driver = agg._fused
    if warmup:
        assert len(driver._flat_all._tapes) == 1 and driver.launches == 1
    else:
        nat = agg._powersgd._native
        assert nat._tapes and all(t.count == nat.launches for t in nat._tapes.values()) and len(nat._tapes) == 2   # one per first side
