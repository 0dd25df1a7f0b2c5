"""The launches that the equality tests of boxes and of the adjoint compare: the pressure
loop's depth shows in its number of box launches, a mask that no box shape allows falls
back, and the staged adjoint step is the staged kernel."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import xgrid
import workloads
from xgrid_gb300 import adjoint, device, runtime
from xgrid_gb300.operator import Operator
from test_gpu_tables_by_iterations import _grids, walled
from test_gpu_tloop import TLOOP_SITE, _sites

pytestmark = pytest.mark.gpu


def _box_launches(k, call):
    return sum(1 for s in _sites(k, call) if s % 64 == TLOOP_SITE)


@pytest.mark.parametrize("n,precision,deep", [(33, "double", True), (131, "double", True), (257, "double", True),
                                              (700, "double", True), (1203, "double", False), (201, "float", False)])
def test_cavity_loop_runs_on_boxes(cacheroot, n, precision, deep):
    xgrid.init(precision=precision, cacheroot=cacheroot, opt_level=3)
    k = Operator(workloads.cavity_kernel.func, "kernel", "cavity_kernel")
    g, cfg = workloads.cavity_setup(n, 5e-6, seed=n)
    args = (g["b"], g["p"], g["u"], g["v"], cfg)
    k(*args)
    depths = {-(-50 // d): d for d in range(2, 7)}
    assert depths[_box_launches(k, lambda: k(*args))] >= (4 if deep else 2)


@pytest.mark.parametrize("wall,iters,launches", [(27, 20, 4), (22, 20, 7), (25, 20, 0), (103, 20, 0), (27, 3, 0),
                                                 (22, 3, 1), (40, 2, 1)])
def test_walls_inside_the_grid(cacheroot, wall, iters, launches):
    """Depth 6 (cores of 20 columns), depth 3 (26 columns) where a wall column on an inner edge
    forbids 6, one launch per iteration where it forbids both."""
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3)
    k = Operator(walled, "kernel", "walled")
    p, f = _grids(150, wall)
    k(p, f, iters)
    assert _box_launches(k, lambda: k(p, f, iters)) == launches


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("shape", [(40, 33, 127), (16, 9, 132)])
def test_adjoint_step_is_the_staged_kernel(cacheroot, precision, shape):
    xgrid.init(precision=precision, cacheroot=cacheroot, opt_level=3, overstep="wrap")
    lib = runtime.load()
    dtype = torch.float32 if precision == "float" else torch.float64
    for staged in (True, False):
        ro = adjoint.Rollout(Operator(workloads.diffuse3d.func, "kernel", "diffuse3d"), 5)
        ro.set_zstage(staged)
        a, b = (torch.rand(shape, dtype=dtype, device="cuda").requires_grad_(True) for _ in range(2))
        lib.xg_prof_reset()
        lib.xg_prof_enable(1)
        try:
            (ro(a, {"k": b}, (0.01,)) ** 2).mean().backward()
            device.stream().synchronize()
            torch.cuda.synchronize()
        finally:
            lib.xg_prof_enable(0)
        sites = [g for g, _ in runtime.prof_records()]
        assert sites.count(-3) == (5 if staged else 0) and sites.count(-2) == (0 if staged else 5)
