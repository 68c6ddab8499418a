"""The tiles that hold a stretch of cells (csrc/hosttiles.h) against those of its
cells one by one, on CPU: axes shorter and longer than a tile, periodic or not,
any halo."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fortran-mpi-fdtd_gb300", "csrc")

DRIVER = r"""
#include <cstdio>
#include <tuple>
#include <vector>
#include "hosttiles.h"
using namespace fdtd;
static unsigned long long s = 12345;
static int rnd(int n) { s = s * 6364136223846793005ull + 1442695040888963407ull; return (int)((s >> 33) % n); }
int main() {
  for (int it = 0; it < 100000; ++it) {
    const int n = 1 + rnd(300), o = 1 + rnd(120), h = rnd(9), len = o + 2 * h, i = rnd(n), c = 1 + rnd(n - i);
    const bool per = rnd(2);
    std::vector<std::tuple<int, int, int, bool>> one, all;  // cell, tile, place, owned
    for (int x = i; x < i + c; ++x) tiles_of(x, n, per, o, h, len, [&](int t, int l, bool own) { one.push_back({x, t, l, own}); });
    stretches_of(i, c, n, per, o, h, len, [&](int t, int skip, int m, int l, int own0, int own1) {
      for (int u = 0; u < m; ++u) all.push_back({i + skip + u, t, l + u, u >= own0 && u < own1});
    });
    int owned = 0;
    for (auto &a : one) owned += std::get<3>(a);
    std::sort(one.begin(), one.end());
    std::sort(all.begin(), all.end());
    if (one != all || owned != c) {
      printf("differ: n=%d per=%d o=%d h=%d i=%d c=%d, owned %d\n", n, per, o, h, i, c, owned);
      return 1;
    }
  }
  printf("ok\n");
  return 0;
}
"""


def test_stretches_match_cells(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src = tmp_path / "tiles.cpp"
    exe = tmp_path / "tiles"
    src.write_text(DRIVER)
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True, timeout=120)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "ok"
