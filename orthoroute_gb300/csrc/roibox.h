// The box around both terminals of an ROI search, whose cells' marks lie in
// shared memory (route.cu).  Plain host/device arithmetic.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define OGR_HD __host__ __device__
#else
#define OGR_HD
#endif

namespace ogr_box {

struct Box {
  int x0, y0;        // its first cell
  int w, h;          // cells
  int row;           // words of a row (16 cells each)
  int words;         // words of all layers; 0: no box
};

// The cells within `reach` of the rectangle of both terminals.
OGR_HD inline Box around(int nx, int ny, int nz, int sx, int sy, int dx, int dy, int reach, int64_t cap) {
  const int ax = sx < dx ? sx : dx, bx = sx < dx ? dx : sx, ay = sy < dy ? sy : dy, by = sy < dy ? dy : sy;
  Box b;
  b.x0 = ax > reach ? ax - reach : 0;
  b.y0 = ay > reach ? ay - reach : 0;
  b.w = (nx - 1 - bx > reach ? bx + reach : nx - 1) - b.x0 + 1;
  b.h = (ny - 1 - by > reach ? by + reach : ny - 1) - b.y0 + 1;
  b.row = (b.w >> 4) + ((b.w & 15) != 0);
  const int64_t plane = (int64_t)b.row * b.h;              // below 2^58
  b.words = plane <= cap && plane * nz <= cap ? (int)(plane * nz) : 0;
  return b;
}

// The box of the deepest search, of at most `depth` steps, whose marks fit in
// cap words (an arc leads at most one cell aside).  Any depth is allowed: from
// the larger side of the lattice on the box is the whole lattice, and a depth
// of 0 or less asks for the terminals' rectangle alone.
OGR_HD inline Box fit(int nx, int ny, int nz, int sx, int sy, int dx, int dy, int depth, int64_t cap) {
  int hi = nx > ny ? nx : ny;
  if (depth < hi) hi = depth > 0 ? depth : 0;
  Box b = around(nx, ny, nz, sx, sy, dx, dy, hi, cap);
  if (b.words) return b;
  b = around(nx, ny, nz, sx, sy, dx, dy, 0, cap);
  if (!b.words) return b;
  int lo = 0;                    // fits; hi does not
  while (hi - lo > 1) {
    const int mid = lo + (hi - lo) / 2;
    const Box m = around(nx, ny, nz, sx, sy, dx, dy, mid, cap);
    if (m.words) { b = m; lo = mid; }
    else hi = mid;
  }
  return b;
}

}  // namespace ogr_box
