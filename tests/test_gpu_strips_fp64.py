"""Strips of FP32 grids whose sweeps compute in FP64 (Python literals are doubles): which grids
take them, and the bits of the tile kernels, with walls and without, ragged and aligned rows."""
import numpy as np
import pytest

import xgrid
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def heat2d(u: xgrid.grid[float, 2], c: float) -> None:
    u[0, 0] = u[0, 0] + c * (u[1, 0] + u[-1, 0] + u[0, 1] + u[0, -1] - 4.0 * u[0, 0])


def cold2d(u: xgrid.grid[float, 2], c: float) -> None:
    u[0, 0] = u[0, 0] + c * (u[1, 0] + u[-1, 0] + u[0, 1] + u[0, -1] - 4.0 * u[0, 0])
    with xgrid.boundary(1):
        u[0, 0] = 0.0


def cold3d(u: xgrid.grid[float, 3], c: float) -> None:
    u[0, 0, 0] = u[0, 0, 0] + c * (u[1, 0, 0] + u[0, -1, 0] + u[0, 0, 1] - 3.0 * u[0, 0, 0])
    with xgrid.boundary(1):
        u[0, 0, 0] = 0.5


@pytest.mark.parametrize("body,shape,strips", [
    (heat2d, (1500, 1500), True), (heat2d, (1024, 4096), True), (heat2d, (2000, 1153), True),
    (cold2d, (1025, 1025), True), (cold2d, (1024, 1024), True), (cold2d, (700, 1537), True),
    (cold3d, (64, 90, 97), True), (cold3d, (63, 90, 97), False), (cold3d, (64, 96, 96), False), (cold3d, (70, 41, 203), True)])
@pytest.mark.parametrize("overstep", ["none", "wrap"])
def test_strips_equal_tiles(cacheroot, overstep, body, shape, strips):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep=overstep)
    got = []
    for on in (True, False):
        k = Operator(body, "kernel", body.__name__)
        rng = np.random.default_rng(17)
        u = xgrid.Grid(shape, float)
        u.now[...] = rng.random(shape).astype(np.float32)
        if body is not heat2d:
            u.boundary = (rng.random(shape) < 0.1).astype(np.int32)
        k(u, 0.15)
        try:
            k.native.set_zstage(on)
            before = k.native.zstage_launches()
            for _ in range(3):
                k(u, 0.15)
            assert (k.native.zstage_launches() > before) == (on and strips)
        finally:
            k.native.set_zstage(True)
        got.append([u.read(i).tobytes() for i in range(u.time)])
    assert got[0] == got[1]
