"""Launch rules (chunks of strips and of the staged z-walk, tile counts): they pick what a
search over every count picks, in a time that a call of one launch does not feel, on
65536-row grids too.  Host code of the header, on the CPU."""
import os
import shutil
import subprocess

import pytest

from xgrid_gb300 import build

HARNESS = r"""
#include "xgrid_gen.cuh"
#include <chrono>
#include <cstdio>
#include <random>
static int64_t strip_all(int64_t A, int64_t strips, int64_t slots) {
  int64_t best = -1, len = A;
  for (int64_t c = 1; c <= (A / 8 > 1 ? A / 8 : 1) && c <= 4096; ++c) {
    const int64_t l = (A + c - 1) / c, chunks = (A + l - 1) / l;
    const int64_t cost = ((strips * chunks + slots - 1) / slots) * (l + 3);
    if (best < 0 || cost < best) best = cost, len = l;
  }
  return len;
}
static int64_t zstage_all(int64_t Z, int64_t ncb, int sms) {
  int64_t best = -1, len = Z;
  for (int64_t c = 1; c <= (Z / 8 > 1 ? Z / 8 : 1) && c <= 4096; ++c) {
    const int64_t l = (Z + c - 1) / c, chunks = (Z + l - 1) / l, n = (ncb * chunks + sms - 1) / sms;
    const int64_t cost = (l + 3) * (n == 1 ? 19 : n == 2 ? 23 : 10 * n);
    if (best < 0 || cost < best) best = cost, len = l;
  }
  return len;
}
static int64_t tiles_all(int64_t len, int64_t per, int64_t slots, int64_t n0, int flat) {
  const int64_t n1 = flat ? n0 : 1, nmax = len / (flat ? 4 : 8);
  int64_t best = -1, count = n0;
  auto cost = [&](int64_t n) { return ((n * per + slots - 1) / slots) * ((len + n - 1) / n + 2); };
  for (int64_t n = n1; n <= nmax && n <= n1 + 256; ++n)
    if (best < 0 || cost(n) < best) best = cost(n), count = n;
  return best < 0 || 10 * cost(n0) <= 11 * best || count > 65535 ? n0 : count;
}
template <typename F> static double us(F f) {
  double best = 1e9;
  for (int r = 0; r < 5; ++r) {
    const auto t = std::chrono::steady_clock::now();
    volatile int64_t sum = 0;
    for (int i = 0; i < 200; ++i) sum = sum + f(i & 1);
    best = std::min(best, std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t).count() / 200);
  }
  return best;
}
int main() {
  std::mt19937_64 g(5);
  auto pick = [&](double hi) { return (int64_t)std::exp(std::uniform_real_distribution<double>(0, std::log(hi))(g)); };
  long wrong = 0;
  for (int i = 0; i < 20000; ++i) {
    const int64_t len = pick(100000), per = pick(20000), sms = 1 + pick(200), slots = sms * (1 + g() % 24);
    wrong += xg_strip_length(len, per, slots) != strip_all(len, per, slots);
    wrong += xg_zstage_length(len, per, (int)sms) != zstage_all(len, per, (int)sms);
    const int flat = g() & 1;
    const int64_t n0 = std::max<int64_t>(1, len / (1 + g() % 64));
    wrong += xg_tile_parts(len, per, slots, n0, flat) != tiles_all(len, per, slots, n0, flat);
  }
  printf("%ld %.3f %.3f\n", wrong, us([](int k) { return xg_strip_length(65536 + k, 1, 152 * 24); }),
         us([](int k) { return strip_all(65536 + k, 1, 152 * 24); }));
  return 0;
}
"""


def test_rules_match_a_full_search(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    build.ensure_runtime()
    src, exe = tmp_path / "h.cu", tmp_path / "h"
    src.write_text(HARNESS)
    subprocess.run([nvcc, *build.ARCH, "-O2", "-std=c++17", "-w", "-I", build.INCLUDE, "-I", build.CSRC, str(src),
                    "-L", build.LIBDIR, "-lxgrid_gb300", "-Xlinker", f"-rpath,{build.LIBDIR}", "-o", str(exe)],
                   check=True, capture_output=True)
    wrong, rule, full = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert int(wrong) == 0
    assert float(rule) < 0.1 * float(full)  # two counts tried instead of 4096
