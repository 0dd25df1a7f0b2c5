"""The two-operation division by a launch constant (``xg_two_op_divisor``): whatever
divisor the host accepts for it gives the IEEE quotient, on random significands and on
the ones whose quotients lie closest to a midpoint of two doubles, where it could fail;
divisors with a failing case are refused.  Runs on the CPU (host code of the header)."""
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
  std::mt19937_64 g(7);
  long two = 0, n = 0, wrong = 0, refused_right = 0, refused = 0;
  auto sig = [&] { return (double)((g() >> 11) | (1ull << 52)); };
  for (int i = 0; i < 6000; ++i) {
    const double d = i < 1000 ? 1.0 + i : (i < 2000 ? -(i - 999) * 0.1 : ldexp(sig(), (int)(g() % 600) - 300));
    const xg_divisor k = xg_make_divisor(d);
    ++n;
    two += k.two;
    long bad = 0;
    for (int j = 0; j < 1500; ++j) {
      double x = sig();
      if (j & 1) {  // the double next to (a midpoint) * d, and its neighbours
        int e;
        const double dn = ldexp(frexp(fabs(d), &e), 53);
        const unsigned __int128 p = ((unsigned __int128)(2 * (uint64_t)sig() + 1)) * (uint64_t)dn;
        x = (double)(uint64_t)(p >> 54) + (double)((int)(j >> 1) % 3 - 1);
      }
      x = ldexp(x, ilogb(d));
      if (fma(x, k.zh, x * k.zl) != x / d) ++bad;
    }
    if (k.two) wrong += bad;
    else { ++refused; refused_right += bad == 0; }
  }
  printf("%ld %ld %ld %ld\n", n, two, wrong, refused);
  const double edge[] = {ldexp(1.1, 1015), ldexp(1.1, -1015), 5e-324, 0.0, INFINITY, NAN};
  for (double d : edge) printf("%d ", xg_make_divisor(d).two);
  return 0;
}
"""


def test_accepted_divisors_give_the_ieee_quotient(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    build.ensure_runtime()
    src, exe = tmp_path / "h.cu", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([nvcc, *build.ARCH, "-O1", "-Xcompiler", "-ffp-contract=off", "-std=c++17", "-w", "-I", build.INCLUDE,
                    "-I", build.CSRC, str(src), "-L", build.LIBDIR, "-lxgrid_gb300", "-Xlinker",
                    f"-rpath,{build.LIBDIR}", "-o", str(exe)], check=True, capture_output=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    n, two, wrong, refused = (int(v) for v in out[0].split())
    assert wrong == 0
    assert two > 0.9 * n and refused == n - two > 0  # most divisors, not all
    # a divisor whose correction term is subnormal, and those without a reciprocal, are refused
    assert out[1].split()[0] == "0" and out[1].split()[2:] == ["0"] * 4
