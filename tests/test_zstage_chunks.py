"""Chunks of the staged z-walk on FP64 grids: the rule picks what a search over every count
picks, and fills the SMs evenly where the extents allow it.  Host code, on the CPU."""
import os
import shutil
import subprocess

import pytest

from xgrid_gb300 import build

HARNESS = r"""
#include "xgrid_gen.cuh"
#include <cstdio>
#include <random>
int main() {
  std::mt19937_64 g(5);
  auto pick = [&](double hi) { return (int64_t)std::exp(std::uniform_real_distribution<double>(0, std::log(hi))(g)); };
  long wrong = 0;
  for (int i = 0; i < 20000; ++i) {
    const int64_t Z = pick(3000), rows = pick(5000), slots = 8 * (1 + pick(200));
    int64_t best = -1, len = Z;
    for (int64_t c = 1; c <= (Z / 4 > 1 ? Z / 4 : 1); ++c) {
      const int64_t l = (Z + c - 1) / c, cost = (2 * ((c * rows + slots - 1) / slots) + 1) * (l + 3);
      if (best < 0 || cost < best) best = cost, len = l;
    }
    wrong += xg_zstage_length_fp64(Z, rows, slots) != len;
  }
  printf("%ld %ld %ld\n", wrong, (long)xg_zstage_length_fp64(256, 64, 152 * 8), (long)xg_zstage_length_fp64(64, 64, 152 * 8));
  return 0;
}
"""


def test_rule_matches_a_full_search(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    build.ensure_runtime()
    src, exe = tmp_path / "h.cu", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([nvcc, *build.ARCH, "-O2", "-std=c++17", "-w", "-I", build.INCLUDE, "-I", build.CSRC, str(src),
                    "-L", build.LIBDIR, "-lxgrid_gb300", "-Xlinker", f"-rpath,{build.LIBDIR}", "-o", str(exe)],
                   check=True, capture_output=True)
    wrong, long_z, short_z = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert wrong == 0
    # 8 blocks a plane on 152 SMs: 19 or 38 chunks fill them evenly (256 planes: 14 or 7 each), and
    # 64 planes are cut down to 4
    assert long_z in (7, 14) and short_z == 4
