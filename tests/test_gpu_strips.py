"""Strip kernels (2-D and 3-D FP32/int32 sweeps) against the tile kernels, bit for bit:
extents that leave partial strips, rows and chunks, every overstep mode, boundary cells in
every position of a 32-column word, in-place sweeps, two loaded grids."""
import numpy as np
import pytest

import xgrid
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def star2d(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * u[0, 0] + b * (u[0, 1] - u[0, -1]) + a * (u[1, 0] + u[-1, 0])


def walled2d(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * u[0, 0] + b * (u[0, 1] + u[-1, 0])
    with xgrid.boundary(1):
        u[0, 0] = b
    with xgrid.boundary(2):
        u[0, 0] = u[0, 0][0] + a


def jacobi2d(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * (u[0, 1][0] + u[0, -1][0]) + b * u[1, 0][0]


def star3d(u: xgrid.grid[float, 3], a: float, b: float) -> None:
    u[0, 0, 0] = a * (u[1, 0, 0] + u[0, 1, 0] + u[0, 0, 1]) - b * (u[-1, 0, 0] + u[0, -1, 0] + u[0, 0, -1])


def walled3d(u: xgrid.grid[float, 3], a: float, b: float) -> None:
    u[0, 0, 0] = a * u[0, 0, 0] + b * (u[0, -1, 0] + u[0, 0, 1] + u[1, 0, 0])
    with xgrid.boundary(1):
        u[0, 0, 0] = b


def inplace3d(u: xgrid.grid[float, 3], a: float, b: float) -> None:
    u[0, 0, 0] = a * (u[1, 0, 0][0] + u[0, 1, 0][0]) + b * u[0, 0, -1][0]


def twogrids3d(u: xgrid.grid[float, 3], a: float, b: float, k: xgrid.grid[float, 3]) -> None:
    u[0, 0, 0] = a * u[0, 0, 0] + b * (k[0, 1, 0] + k[0, 0, -1]) * (u[0, 0, 1] - u[-1, 0, 0])


def ints2d(u: xgrid.grid[int, 2], a: int, b: int) -> None:
    u[0, 0] = a * u[0, 1] + b * u[0, -1] - u[1, 0] + u[-1, 0]


CASES = [(star2d, (2051, 1025)), (star2d, (700, 3071)), (walled2d, (1100, 1000)), (jacobi2d, (1511, 1513)),
         (star3d, (37, 61, 129)), (star3d, (9, 3, 8191)), (star3d, (33, 70, 250)), (walled3d, (65, 90, 97)),
         (walled3d, (40, 70, 225)), (inplace3d, (40, 67, 63)), (inplace3d, (20, 40, 200)), (twogrids3d, (35, 65, 131)),
         (ints2d, (1400, 1603))]


@pytest.mark.parametrize("overstep", ["none", "limit", "wrap"])
@pytest.mark.parametrize("body,shape", CASES, ids=[f"{f.__name__}-{'x'.join(map(str, s))}" for f, s in CASES])
def test_strips_equal_tiles(cacheroot, overstep, body, shape):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep=overstep)
    element = int if body is ints2d else float
    got = []
    for strips in (True, False):
        k = Operator(body, "kernel", body.__name__)
        rng = np.random.default_rng(17)
        u = xgrid.Grid(shape, element)
        extra = (xgrid.Grid(shape, element),) if body is twogrids3d else ()
        for g in (u, *extra):
            g.now[...] = rng.integers(-9, 9, shape) if element is int else rng.random(shape).astype(np.float32)
        if body in (walled2d, walled3d, jacobi2d, inplace3d):
            u.boundary = (rng.random(shape) < 0.1).astype(np.int32) * rng.integers(1, 3, shape).astype(np.int32)
        values = (3, -2) if element is int else (0.3, 0.2)
        k(u, *values, *extra)  # compiles
        k.native.set_zstage(strips)
        before = k.native.zstage_launches()
        for _ in range(3):
            k(u, *values, *extra)
        assert (k.native.zstage_launches() > before) == strips
        got.append([u.read(i) for i in range(u.time)])
    for a, b in zip(*got):
        assert a.tobytes() == b.tobytes()
