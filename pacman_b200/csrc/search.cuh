// Nearest-neighbour scan of a uniform cell grid, shared by nearest.cu and
// mls.cu: shells of cells around the query's cell, nearest first, until no
// unscanned cell can hold a closer source.
#pragma once

#include "common.cuh"

namespace pacman_b200 {

// Distance from y to the nearest face of the scanned block of cells (shells
// 0..R around cell c) behind which unscanned cells lie; infinity if there are
// none.  Every unscanned source is at least that far away, less the rounding
// of the cell assignment, which scan_shells covers with a millionth of a cell
// (the assignment's error is below 2^-23 cells for 2^28 cells per axis).
template <int DIM>
__device__ __forceinline__ double scanned_reach(const GridView &g, const double *y, const int *c,
                                                int R, double h) {
  double reach = INFINITY;
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    if (c[d] - R > 0) reach = fmin(reach, y[d] - (g.lo[d] + double(c[d] - R) * h));
    if (c[d] + R + 1 < g.nc[d]) reach = fmin(reach, (g.lo[d] + double(c[d] + R + 1) * h) - y[d]);
  }
  return reach;
}

__device__ __forceinline__ bool has_nan(const double4 &q) {
  return isnan(q.x) || isnan(q.y) || isnan(q.z);
}

// Calls visit(point) for the cell-sorted sources shell by shell; after each
// shell worst() is the squared distance that a further source would have to
// beat (infinity while fewer than wanted are known).  Not for a query with a NaN
// coordinate (has_nan), which would visit every cell and find nothing.
template <int DIM, typename Visit, typename Worst>
__device__ __forceinline__ void scan_shells(const GridView &g, const double4 *__restrict__ sorted,
                                            double h, const double4 &q, Visit &&visit,
                                            Worst &&worst) {
  const double y[3] = {q.x, q.y, q.z};
  const int c[3] = {cell_coord(q.x, g.lo[0], g.inv_h, g.nc[0]),
                    DIM > 1 ? cell_coord(q.y, g.lo[1], g.inv_h, g.nc[1]) : 0,
                    DIM > 2 ? cell_coord(q.z, g.lo[2], g.inv_h, g.nc[2]) : 0};
  auto scan = [&](int s, int e) {
    for (int i = s; i < e; ++i) visit(sorted[i]);
  };
  for (int R = 0;; ++R) {
    const int x0 = max(c[0] - R, 0), x1 = min(c[0] + R, g.nc[0] - 1);
    const int y0 = max(c[1] - R, 0), y1 = min(c[1] + R, g.nc[1] - 1);
    const int z0 = max(c[2] - R, 0), z1 = min(c[2] + R, g.nc[2] - 1);
    for (int a = x0; a <= x1; ++a)
      for (int b = y0; b <= y1; ++b) {
        const int base = (a * g.nc[1] + b) * g.nc[2];
        const bool face = a == c[0] - R || a == c[0] + R || b == c[1] - R || b == c[1] + R;
        if (face) {  // the whole z run of this column is on the shell
          scan(g.start[base + z0], g.start[base + z1 + 1]);
        } else {  // only its two ends
          if (c[2] - R >= 0) scan(g.start[base + c[2] - R], g.start[base + c[2] - R + 1]);
          if (c[2] + R < g.nc[2]) scan(g.start[base + c[2] + R], g.start[base + c[2] + R + 1]);
        }
      }
    const bool all = c[0] - R <= 0 && c[0] + R >= g.nc[0] - 1 && c[1] - R <= 0 &&
                     c[1] + R >= g.nc[1] - 1 && c[2] - R <= 0 && c[2] + R >= g.nc[2] - 1;
    if (all) return;
    const double lim = scanned_reach<DIM>(g, y, c, R, h) - 1e-6 * h;
    if (lim > 0.0 && worst() < lim * lim) return;
  }
}

}  // namespace pacman_b200
