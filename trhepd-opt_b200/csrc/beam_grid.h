// The index grid of a beam set (host side).
#pragma once
#include <algorithm>
#include <cstdlib>
#include <vector>

namespace trhepd {

// Beams on a grid: the stage matrix V(k, j) depends on the difference of beams k and j
// only, so Q V is a convolution over the grid of the beams' (transformed) indices.
// Beam j sits at (x, y), 0 <= x < sx, 0 <= y < sy; transforms have length m >= sx, sy
// and two parities per dimension (2 m points).
struct ConvGrid {
  int m = 0;                   // 0: the beams have no such grid (or it does not pay)
  int sx = 0, sy = 0;
  std::vector<int> cell;       // beam -> y << 8 | x
  std::vector<unsigned> mask;  // line y: bit x set where a beam sits
  // table entry of each difference: cell (dy mod 2m) * 2m + (dx mod 2m) holds 0 (none),
  // e + 1 (-conj(u[e])) or -(e + 1) (-w[e])
  std::vector<int> entry;
  // (e1, e2) pairs that must satisfy conj(u[e1]) = w[e2] in every column: a difference
  // met in both beam orders
  std::vector<int> twins;
};

// pair: the n x n beam-pair map (0-based table indices).  An empty grid (m = 0) where the
// map is not a function of the beam difference, the span is beyond 32 or the grid is too
// sparse to pay.
inline ConvGrid conv_grid(int n, const int* ih, const int* ik, const int* pair) {
  ConvGrid g;
  if (n <= 64) return g;  // below, the dense products are as cheap (and fused, small.cu)
  // beam indices relative to beam 0, sheared to the smallest bounding grid
  int best = 1 << 30, shear = 0, axis = 0;
  auto span = [&](int c, int ax, int& sx, int& sy, int& x0, int& y0) {
    int x1, y1;
    x0 = y0 = 1 << 29;
    x1 = y1 = -(1 << 29);
    for (int j = 0; j < n; ++j) {
      const int x = ax ? ih[j] + c * ik[j] : ih[j], y = ax ? ik[j] : ik[j] + c * ih[j];
      x0 = std::min(x0, x);
      x1 = std::max(x1, x);
      y0 = std::min(y0, y);
      y1 = std::max(y1, y);
    }
    sx = std::min(x1 - x0, 1 << 15) + 1;
    sy = std::min(y1 - y0, 1 << 15) + 1;
  };
  for (int j = 0; j < n; ++j)
    if (std::abs(ih[j]) > (1 << 20) || std::abs(ik[j]) > (1 << 20)) return g;
  for (int ax = 0; ax < 2; ++ax)
    for (int c = -2; c <= 2; ++c) {
      int sx, sy, x0, y0;
      span(c, ax, sx, sy, x0, y0);
      const int key = std::max(sx, sy) * 4096 + std::min(sx, sy);
      if (key < best) {
        best = key;
        shear = c;
        axis = ax;
      }
    }
  int sx, sy, x0, y0;
  span(shear, axis, sx, sy, x0, y0);
  int m = 0;
  for (int l : {9, 10, 12, 15, 16, 20, 25, 27, 32})
    if (l >= std::max(sx, sy)) {
      m = l;
      break;
    }
  // Below this filling the dense FP64 product may be as fast.  Thin-slice solves, us per
  // stage, convolution / dense, 61 angles (m >= 25: 31): at the line m = 15, n = 92 28 / 50,
  // m = 20, n = 162 95 / 145, m = 25, n = 252 159 / 199, m = 27, n = 293 195 / 341; at a
  // filling of 0.32 (74 beams) 23 / 32, (130) 75 / 109, (202) 128 / 159, (235) 154 / 184; of
  // 0.25 (102) 61 / 57, (158) 99 / 71, (184) 121 / 84.
  if (!m || (double)n < 0.4 * m * m) return g;
  g.sx = sx;
  g.sy = sy;
  g.cell.resize(n);
  g.mask.assign(sy, 0u);
  std::vector<int> px(n), py(n);
  for (int j = 0; j < n; ++j) {
    px[j] = (axis ? ih[j] + shear * ik[j] : ih[j]) - x0;
    py[j] = (axis ? ik[j] : ik[j] + shear * ih[j]) - y0;
    if ((g.mask[py[j]] >> px[j]) & 1u) return ConvGrid{};  // two beams in one cell
    g.mask[py[j]] |= 1u << px[j];
    g.cell[j] = py[j] << 8 | px[j];
  }
  const int L = 2 * m;
  std::vector<int> up((size_t)L * L, 0), dn((size_t)L * L, 0);
  up[0] = 1;  // the diagonal: -conj(u[0])
  for (int k = 0; k < n; ++k)
    for (int j = 0; j < n; ++j) {
      if (j == k) continue;
      const int c = ((py[j] - py[k] + L) % L) * L + (px[j] - px[k] + L) % L;
      int& slot = (k < j ? up : dn)[c];
      const int e = pair[(size_t)k * n + j] + 1;
      if (slot == 0) slot = e;
      else if (slot != e) return ConvGrid{};  // not a function of the difference
    }
  g.entry.assign((size_t)L * L, 0);
  for (int c = 0; c < L * L; ++c) {
    g.entry[c] = up[c] ? up[c] : -dn[c];
    if (up[c] && dn[c]) {
      g.twins.push_back(up[c] - 1);
      g.twins.push_back(dn[c] - 1);
    }
  }
  g.m = m;
  return g;
}

}  // namespace trhepd
