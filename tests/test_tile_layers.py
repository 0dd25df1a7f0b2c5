"""Layers of tiles along z of 3-D tile launches: close to the least cost over every count, never
fewer than 4 planes a tile, and more than one round where remainder tiles take longer.  Host
code of the header, on the CPU; the same bits for any count, on the GPU."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import xgrid
from xgrid_gb300 import build
from xgrid_gb300.operator import Operator

HARNESS = r"""
#include "xgrid_gen.cuh"
#include <cstdio>
#include <random>
int main() {
  std::mt19937_64 g(5);
  auto pick = [&](double hi) { return (int64_t)std::exp(std::uniform_real_distribution<double>(0, std::log(hi))(g)); };
  double worst = 0;
  long bad = 0;
  for (int i = 0; i < 5000; ++i) {
    const int64_t len = pick(3000), work = pick(30000), longest = 1 + (int64_t)(g() % 4), slots = 152 * (4 + g() % 3);
    const int64_t hi = len / 4 > 1 ? len / 4 : 1, n = xg_tile_parts_3d(len, slots, work, longest);
    auto cost = [&](int64_t k) {
      const int64_t whole = (k * work + slots - 1) / slots, part = (len + k - 1) / k;
      return (0.5 * whole + 0.5 * (double)(k * work) / slots + 0.5 * longest) * (part + 1);
    };
    double best = cost(1);
    for (int64_t k = 2; k <= hi; ++k) best = std::min(best, cost(k));
    bad += n < 1 || n > hi;
    worst = std::max(worst, cost(n) / best);
  }
  printf("%ld %.3f %ld\n", bad, worst, (long)xg_tile_parts_3d(300, 152 * 6, 375, 2));
  return 0;
}
"""


def test_rule_is_close_to_a_full_search(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    build.ensure_runtime()
    src, exe = tmp_path / "h.cu", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([nvcc, *build.ARCH, "-O2", "-std=c++17", "-w", "-I", build.INCLUDE, "-I", build.CSRC, str(src),
                    "-L", build.LIBDIR, "-lxgrid_gb300", "-Xlinker", f"-rpath,{build.LIBDIR}", "-o", str(exe)],
                   check=True, capture_output=True)
    bad, worst, ragged = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert int(bad) == 0 and float(worst) < 1.25
    assert int(ragged) >= 12  # a 300^3 grid: 3 layers filled one round of CTAs


def diag3d(u: xgrid.grid[float, 3], a: float, b: float) -> None:
    u[0, 0, 0] = a * (u[1, 1, 0] + u[0, 1, 1]) + b * (u[-1, -1, 0] + u[-1, 0, -1] + u[0, 0, 0])
    with xgrid.boundary(1):
        u[0, 0, 0] = a * u[1, 0, 0][0]


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(33, 37, 70), (4, 9, 64), (3, 64, 129), (1, 50, 200), (64, 5, 65), (100, 3, 300), (29, 64, 63)])
@pytest.mark.parametrize("overstep", ["none", "wrap"])
def test_layers_keep_the_bits(cacheroot, shape, overstep):
    xgrid.init(precision="double", cacheroot=cacheroot, opt_level=3, overstep=overstep)
    k = Operator(diag3d, "kernel", "diag3d")
    out = []
    for tiling in (None, (64, 4, 64, 64, 4, 1), (-1, 4, 64, 64, 4, 1)):
        rng = np.random.default_rng(3)
        u = xgrid.Grid(shape, float)
        u.now[...] = rng.random(shape)
        u.boundary[0] = 1
        k(u, 0.2, 0.1)
        try:
            k.native.set_tiling(0, tiling)
            for _ in range(3):
                k(u, 0.2, 0.1)
        finally:
            k.native.set_tiling(0, None)
        out.append([u.read(i).tobytes() for i in range(u.time)])
    assert out[0] == out[1] == out[2]
