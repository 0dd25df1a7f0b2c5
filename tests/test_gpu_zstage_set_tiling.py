"""A set tiling keeps mask-free 3-D sweeps of unaligned rows on the staged z-walk, also
where an untuned sweep takes strips: same bits as tiles and strips."""
import numpy as np
import pytest

import xgrid
import workloads
from xgrid_gb300.operator import Operator

pytestmark = pytest.mark.gpu


def star3d(u: xgrid.grid[float, 3], a: float, b: float) -> None:
    u[0, 0, 0] = a * (u[1, 0, 0] + u[0, 1, 0] + u[0, 0, 1]) - b * (u[-1, 0, 0] + u[0, -1, 0] + u[0, 0, -1])


@pytest.mark.parametrize("overstep", ["wrap", "limit"])
@pytest.mark.parametrize("program", ["star3d", "diffuse3d"])
@pytest.mark.parametrize("shape", [(40, 70, 225), (37, 40, 70), (9, 33, 35), (64, 64, 65), (17, 9, 131)])
def test_unaligned_rows_stay_staged(cacheroot, overstep, program, shape):
    xgrid.init(precision="float", cacheroot=cacheroot, opt_level=3, overstep=overstep)
    body, values = (star3d, (0.3, 0.2)) if program == "star3d" else (workloads.diffuse3d.func, (0.05,))
    got = []
    for how in ("staged", "untuned", "tiles"):
        k = Operator(body, "kernel", program)
        rng = np.random.default_rng(17)
        grids = [xgrid.Grid(shape, float) for _ in range(2 if program == "diffuse3d" else 1)]
        for g in grids:
            g.now[...] = rng.uniform(0.01, 0.1, shape).astype(np.float32)
        k(*grids, *values)
        nk = k.native
        try:
            nk.set_zstage(how != "tiles")
            if how != "untuned":
                nk.set_tiling(0, (64, 4, 64, 64, 4, 1))
            before = nk.zstage_launches()
            for _ in range(3):
                k(*grids, *values)
            if how != "untuned":
                assert (nk.zstage_launches() > before) == (how == "staged")
        finally:
            nk.set_zstage(True)
            nk.set_tiling(0, None)
        got.append([grids[0].read(i).tobytes() for i in range(grids[0].time)])
    assert got[0] == got[1] == got[2]
