"""Strips hold column numbers in 32 bits: rows whose last strip or its neighbour column would
not fit keep the tiles.  The generated rule alone, as host code on the CPU (such a grid takes
17 GB)."""
import re
import shutil
import subprocess

import pytest

import xgrid
from xgrid_gb300 import build
from xgrid_gb300.codegen import CudaGenerator
from xgrid_gb300.config import get_config
from xgrid_gb300.operator import Operator


def star2d(u: xgrid.grid[float, 2], a: float) -> None:
    u[0, 0] = a * u[0, 0] + a * (u[0, 1] - u[0, -1])


def star3d(u: xgrid.grid[float, 3], a: float) -> None:
    u[0, 0, 0] = a * u[0, 0, 1] + a * (u[0, 1, 0] - u[-1, 0, 0])


@pytest.mark.parametrize("body,tail", [(star2d, "{1, X}"), (star3d, "{1, 9, X}")])
def test_rows_beyond_int_columns_keep_the_tiles(tmp_path, body, tail):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    xgrid.init(precision="float", cacheroot=str(tmp_path), opt_level=3, overstep="wrap")
    n = body.__name__
    text = CudaGenerator(Operator(body, "kernel", n), get_config()).generate().source
    rule = re.search(rf"static int xgl_{n}_0_strips\(const xg_grid\* G\) \{{.*?\n\}}", text, re.S).group(0)
    header = open(build.CSRC + "/xgrid_gen.cuh").read()
    extent = "\n".join(re.search(pat, header, re.S).group(0) for pat in
                       (r"struct xg_ext \{[^}]*\};", r"static inline xg_ext xg_extent\(.*?\n\}",
                        r"static inline bool xg_same_ext\([^}]*\}"))
    src, exe = tmp_path / "h.cpp", tmp_path / "h"
    src.write_text(f"""#include "xgrid_gb300.h"
#include <cstdio>
#include <initializer_list>
{extent}
static int xg_zstage_{n} = 1;
static unsigned char xg_tiling_set_{n}[1];
{rule}
int main() {{
  for (int64_t X : {{(int64_t)1 << 22, ((int64_t)1 << 30) - 1, ((int64_t)1 << 31) - 1, ((int64_t)1 << 31) + 100,
                    ((int64_t)1 << 32) + 128}}) {{
    xg_grid g{{}};
    g.ndim = {tail.count(',') + 1};
    const int64_t shape[] = {tail};
    for (int i = 0; i < g.ndim; ++i) g.shape[i] = shape[i];
    printf("%d ", xgl_{n}_0_strips(&g) != 0);
  }}
  return 0;
}}
""")
    subprocess.run(["g++", "-std=c++17", "-I", build.INCLUDE, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split() == ["1", "1", "0", "0", "0"]
