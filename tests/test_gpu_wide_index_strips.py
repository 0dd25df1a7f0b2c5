"""64-bit indices on the strip kernels and the batched kernels: grids above the strips' floors
and batches, run with ``xg_force_wide_index`` on, give the bits of the 32-bit kernels."""
import numpy as np
import pytest

import xgrid
import workloads
from xgrid_gb300 import native, runtime
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def star2d(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * u[0, 0] + b * (u[0, 1] - u[0, -1]) + a * (u[1, 0] + u[-1, 0])
    with xgrid.boundary(1):
        u[0, 0] = b


def star3d(u: xgrid.grid[float, 3], a: float, b: float) -> None:
    u[0, 0, 0] = a * (u[1, 0, 0] + u[0, 1, 0] + u[0, 0, 1]) - b * (u[-1, 0, 0] + u[0, -1, 0] + u[0, 0, -1])
    with xgrid.boundary(1):
        u[0, 0, 0] = b


def jacobi2d(u: xgrid.grid[float, 2], a: float, b: float) -> None:
    u[0, 0] = a * (u[0, 1][0] + u[0, -1][0]) + b * u[1, 0][0]


def _wide(run):
    lib = runtime.load()
    out = []
    try:
        for wide in (0, 1):
            lib.xg_force_wide_index(wide)
            lib.xg_graph_clear(None)
            out.append(run())
    finally:
        lib.xg_force_wide_index(0)
        lib.xg_graph_clear(None)
    return out


@pytest.mark.parametrize("overstep", ["none", "limit", "wrap"])
@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("body,shape", [(star2d, (1511, 1513)), (jacobi2d, (1511, 1513)), (star3d, (65, 90, 97)),
                                        (star3d, (40, 70, 225))])
def test_strips(cacheroot, overstep, masked, body, shape):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep=overstep)

    def run():
        k = Operator(body, "kernel", f"{body.__name__}_ws")
        rng = np.random.default_rng(5)
        u = xgrid.Grid(shape, float)
        u.now[...] = rng.random(shape).astype(np.float32)
        if masked:
            u.boundary = (rng.random(shape) < 0.1).astype(np.int32)
        k(u, 0.3, 0.2)
        before = k.native.zstage_launches()
        for _ in range(3):
            k(u, 0.3, 0.2)
        assert k.native.zstage_launches() > before
        return [u.read(i).tobytes() for i in range(u.time)]
    a, b = _wide(run)
    assert a == b


@pytest.mark.parametrize("temporal", [1, (6, 52, 116), (12, 104, 104)])
@pytest.mark.parametrize("precision", ["float", "double"])
def test_batch(cacheroot, monkeypatch, precision, temporal):
    if precision == "double" and temporal == (12, 104, 104):
        pytest.skip("the box does not fit a CTA's shared memory")
    xgrid.init(precision=precision, cacheroot=cacheroot, opt_level=3, overstep="wrap")
    small = []
    for name, at in (("BatchArgs", 7), ("BatchTemporalArgs", 5)):
        real = getattr(native, name)
        monkeypatch.setattr(native, name, lambda *a, real=real, at=at: small.append(a[at]) or real(*a))

    def run():
        k = Operator(workloads.convdiff2d.func, "kernel", "convdiff2d")
        rng = np.random.default_rng(21)
        out = []
        for shape in [(14, 131), (64, 128), (105, 58), (53, 233)]:
            g = xgrid.Grid(shape, float)
            g.now[...] = rng.random(shape)
            out.append((g, *(float(v) for v in rng.uniform(0.01, 0.2, 5))))
        for _ in range(2):
            k.batch(out, 13, temporal=temporal)
        return [p[0].read(i).tobytes() for p in out for i in (0, 1)]
    a, b = _wide(run)
    assert a == b
    assert small == [1, 1, 0, 0]
