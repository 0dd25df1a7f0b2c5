"""Tuner candidates of batched time loops by the kernel that runs them: low tiles for programs
in shared memory alone (FP64 fields, two-cell reach), boxes of 128 x 128 for register blocks."""
import pytest

import xgrid
import workloads
from xgrid_gb300 import autotune
from xgrid_gb300.codegen import CudaGenerator
from xgrid_gb300.config import get_config
from xgrid_gb300.operator import Operator


def wide(u: xgrid.grid[float, 2], a: float) -> None:
    u[0, 0] = u[0, 0] + a * (u[0, 2] + u[-2, 0])


@pytest.mark.parametrize("body,precision,registers", [(workloads.convdiff2d.func, "float", True),
                                                      (workloads.convdiff2d.func, "double", False),
                                                      (wide, "float", False), (wide, "double", False)])
def test_candidates_by_kernel(body, precision, registers):
    xgrid.init(precision=precision, overstep="wrap")
    m = CudaGenerator(Operator(body, "kernel", body.__name__), get_config()).generate()
    assert m.batch and m.batch_registers == registers
    out = autotune.batch_candidates(False, m.batch_registers)
    assert ((2, 16, 60, (32, 8, 1)) in out) != registers
    assert ((2, 124, 124, (32, 8, 1)) in out) == registers
    assert len(out) == len(set(out)) and all(autotune.TUNE_STEPS % c[0] == 0 for c in out)
    if not registers:  # every tile and its halo fit a CTA's shared memory
        r, size = (2 if body is wide else 1), (8 if precision == "double" else 4)
        assert all(2 * size * (ty + 2 * d * r) * (tx + 2 * d * r) < 232448 for d, ty, tx, _ in out)
