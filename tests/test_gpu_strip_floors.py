"""Smallest grids on strips by the boundary phases of the sweep: groups of three and more stay
one fused launch on rows of whole tiles up to twice the cells.  Same bits either way."""
import numpy as np
import pytest

import xgrid
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def walls2(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * u[0, 0] + b * (u[0, 1] + u[0, -1] + u[1, 0] + u[-1, 0])
    with xgrid.boundary(1):
        u[0, 0] = b
    with xgrid.boundary(2):
        u[0, 0] = a


def walls3(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * u[0, 0] + b * (u[0, 1] + u[0, -1] + u[1, 0] + u[-1, 0])
    with xgrid.boundary(1):
        u[0, 0] = b
    with xgrid.boundary(2):
        u[0, 0] = a
    with xgrid.boundary(3):
        u[0, 0] = u[1, 0][0]


@pytest.mark.parametrize("body,shape,strips", [
    (walls2, (1024, 1024), True), (walls2, (1023, 1024), False), (walls3, (1024, 1024), False),
    (walls3, (2047, 1024), False), (walls3, (2048, 1024), True), (walls3, (1030, 1025), True), (walls3, (1020, 1025), False)])
def test_floor_by_phases(cacheroot, body, shape, strips):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3)
    got = []
    for on in (True, False):
        k = Operator(body, "kernel", body.__name__)
        u = xgrid.Grid(shape, float)
        u.now[...] = np.random.default_rng(2).random(shape)
        u.boundary[:, 0] = u.boundary[:, -1] = 1
        u.boundary[-1, :] = 2
        u.boundary[0, :] = 3 if body is walls3 else 2
        k(u, 0.2, 0.15)
        nk = k.native
        try:
            nk.set_zstage(on)
            before = nk.zstage_launches()
            for _ in range(3):
                k(u, 0.2, 0.15)
            assert (nk.zstage_launches() > before) == (on and strips)
        finally:
            nk.set_zstage(True)
        got.append([u.read(i).tobytes() for i in range(u.time)])
    assert got[0] == got[1]
