// The overlapping tiles of an axis that hold a cell or a stretch of cells, for the
// block-step kernels' tables.  Plain C++, no CUDA: the CPU tests compile it on its
// own.
#pragma once

#include <algorithm>

namespace fdtd {

// The tiles of width `len` (o cells owned, h of halo) that hold cell i of an
// axis of n cells: calls f(tile, place in the tile, whether the tile owns it).
// On a periodic axis the halo wraps, so a tile may hold images of a cell.
template <typename F>
void tiles_of(int i, int n, bool per, int o, int h, int len, F f) {
  const int nt = (n + o - 1) / o;
  const int lo = -h, hi = (nt - 1) * o - h + len;  // the span of all tiles
  const int m0 = per ? -((i - lo) / n) : 0, m1 = per ? (hi - 1 - i) / n : 0;
  for (int m = m0; m <= m1; ++m) {
    const int x = i + m * n;
    if (x < lo || x >= hi) continue;
    const int t0 = std::max(0, (x + h - len + 1 + o - 1) / o), t1 = std::min(nt - 1, (x + h) / o);
    for (int t = t0; t <= t1; ++t) {
      const int l = x - (t * o - h);
      if (l >= 0 && l < len) f(t, l, m == 0 && l >= h && l < h + o);
    }
  }
}

// The same of the cells i .. i+count-1: f(tile, cells before the stretch, its
// length, place of its first cell, from which to which of its cells are owned)
template <typename F>
void stretches_of(int i, int count, int n, bool per, int o, int h, int len, F f) {
  const int nt = (n + o - 1) / o;
  const int lo = -h, hi = (nt - 1) * o - h + len;
  const int m0 = per ? -((i + count - 1 - lo) / n) : 0, m1 = per ? (hi - 1 - i) / n : 0;
  for (int m = m0; m <= m1; ++m) {
    const int x0 = std::max(i + m * n, lo), x1 = std::min(i + count + m * n, hi);
    if (x0 >= x1) continue;
    const int t0 = std::max(0, (x0 + h - len + 1 + o - 1) / o), t1 = std::min(nt - 1, (x1 - 1 + h) / o);
    for (int t = t0; t <= t1; ++t) {
      const int b = t * o - h, a0 = std::max(x0, b), a1 = std::min(x1, b + len);
      if (a0 >= a1) continue;
      const int w0 = std::max(a0, b + h), w1 = std::min(a1, b + h + o);
      f(t, a0 - (i + m * n), a1 - a0, a0 - b, m == 0 ? w0 - a0 : 0, m == 0 ? std::max(w0, w1) - a0 : 0);
    }
  }
}

}  // namespace fdtd
