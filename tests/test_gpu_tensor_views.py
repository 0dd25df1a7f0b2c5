"""``Grid.tensor``: the tensor of a level's buffer survives calls and level rotation, shows
what the kernel wrote, and is made anew when the caller has changed what it is; a call that
is one launch gives the same bits eager, captured and launched directly afterwards."""
import gc

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import xgrid
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def relax(u: xgrid.grid[float, 2], c: float) -> None:
    u[0, 0] = u[0, 0] + c * (u[0, 1] + u[0, -1] - u[0, 0] - u[0, 0])


@pytest.mark.parametrize("change", [lambda t: t.t_(), lambda t: t.unsqueeze_(0), lambda t: t.requires_grad_(True),
                                    lambda t: t.resize_(3)])
def test_changed_tensors_are_made_anew(cacheroot, change):
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3, overstep="wrap")
    u = xgrid.Grid((8, 8), float)
    x = torch.arange(64, dtype=torch.float64, device="cuda").view(8, 8)
    t = u.tensor(0)
    torch.cuda.synchronize()
    t.copy_(x)
    assert u.tensor(0) is t
    change(t)
    fresh = u.tensor(0)
    assert fresh is not t and fresh.shape == (8, 8) and not fresh.requires_grad
    assert torch.equal(fresh, x)


def test_direct_calls_and_tensors_follow_the_levels(cacheroot):
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3, overstep="wrap")
    k = Operator(relax, "kernel", "relax")
    u = xgrid.Grid((33, 47), float)
    x = np.random.default_rng(3).random((33, 47))
    u.now[...] = x
    for i in range(7):  # eager, captured, then direct, on both rotations of the levels
        k(u, 0.2)
        x = x + 0.2 * (np.roll(x, -1, 1) + np.roll(x, 1, 1) - x - x)
        torch.cuda.synchronize()
        assert np.array_equal(u.tensor(0).cpu().numpy(), x), i


def test_dropped_grids_give_their_memory_back():
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    gc.disable()
    try:
        for _ in range(3):
            u = xgrid.Grid((512, 512), float)
            u.tensor(0)
            del u
        assert torch.cuda.memory_allocated() == before  # no reference cycle through the tensor
    finally:
        gc.enable()
