"""Register z-walk of sweeps that look one way along z only: the window's next plane is the
next plane, whichever of z - 1 and z + 1 the sweep loads (grids with boundary cells, and
mask-free grids with the streaming paths off), against numpy."""
import numpy as np
import pytest

import xgrid
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def down(u: xgrid.grid[float, 3], a: float) -> None:
    u[0, 0, 0] = u[0, 0, 0] + a * u[-1, 0, 0] + a * u[0, 1, 0]


def up(u: xgrid.grid[float, 3], a: float) -> None:
    u[0, 0, 0] = u[0, 0, 0] + a * u[1, 0, 0] + a * u[0, 1, 0]


@pytest.mark.parametrize("body,dz", [(down, 1), (up, -1)])
@pytest.mark.parametrize("masked", [False, True])
def test_one_sided_sweeps(cacheroot, body, dz, masked):
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3, overstep="wrap")
    k = Operator(body, "kernel", f"onesided_{body.__name__}")
    shape = (71, 9, 66)
    x = np.random.default_rng(1).random(shape)
    u = xgrid.Grid(shape, float)
    u.now[...] = x
    if masked:
        u.boundary[70, 8, 65] = 1
    k(u, 0.25)
    y = x + 0.25 * np.roll(x, dz, 0) + 0.25 * np.roll(x, -1, 1)
    if not masked:
        assert np.array_equal(u.read(0), y)
        k.native.set_zstage(False)
        u.now[...] = x
        k(u, 0.25)
    else:
        y[70, 8, 65] = 0.0  # the new level starts from zeros and the sweep leaves the cell alone
    assert np.array_equal(u.read(0), y)
