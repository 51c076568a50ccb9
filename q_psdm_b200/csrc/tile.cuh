// tile.cuh -- what is decided once for an image tile: table coverage and the
// bound of the dip test, shared by the imaging kernels.
#pragma once

#include "common.cuh"

namespace qpsdm {

// The surface-grid test of every table lookup: fractional node coordinates
// of (px, py) in a grid of nxs x nys nodes at spacing 1/rdx, 1/rdy centred
// on (xc, 0), and whether they lie inside it.  Explicit IEEE operations (the
// oracle repeats them bit for bit), because a pair is evaluated -- and
// counted as a point-trace -- exactly when both its lookups pass this test.
__device__ __forceinline__ bool grid_pos(float px, float py, float xc, float rdx, float rdy,
                                         float hx, float hy, int nxs, int nys, float &fx,
                                         float &fy) {
  fx = __fmaf_rn(__fsub_rn(px, xc), rdx, hx);
  fy = __fmaf_rn(py, rdy, hy);
  return fx >= 0.0f && fx <= (float)(nxs - 1) && fy >= 0.0f && fy <= (float)(nys - 1);
}

// Tile-level dip test.  A member (source S, receiver G) contributes to an
// image point P only if the bisector u = A_S + A_G of the unit vectors from
// P passes the four division-free dip tests
//   fx1 = ux - tanx1c uz > 0,  fx2 = tanx2c uz - ux > 0   (y likewise),
// so it can be dropped for a whole image tile when an upper bound of one of
// them over the tile is negative.  The bounds come from interval arithmetic
// over the tile's box (x in [x0, x1], y = 0 on the line, z in [z0, z1]) and
// the tile's ranges of the four dip limits; the margin 1e-4 max(1, |tan|)
// (|tan| the largest dip-limit tangent of the tile: the test functions'
// rounding grows with tan uz) covers the FP32 rounding of the per-point test,
// so no member that passes at some point of the tile is dropped (the kernel's
// sums are unchanged).
struct TileBox {
  float x0, x1, z0, z1;
  float t1lo, t1hi, t2lo, t2hi, u1lo, u1hi, u2lo, u2hi;  // tanx1c, tanx2c, tany1c, tany2c
  float margin;  // -1e-4 max(1, largest |tan| of the tile)
};
struct UnitBounds {
  float axl, axh, ayl, ayh, azl, azh;
  bool ok;
};
__device__ __forceinline__ UnitBounds unit_bounds(float px, float py, const TileBox &b) {
  UnitBounds u;
  const float dxl = px - b.x1, dxh = px - b.x0;
  const float adxmin = (dxl <= 0.0f && dxh >= 0.0f) ? 0.0f : fminf(fabsf(dxl), fabsf(dxh));
  const float adxmax = fmaxf(fabsf(dxl), fabsf(dxh));
  const float rmin2 = adxmin * adxmin + py * py + b.z0 * b.z0;
  const float rmax2 = adxmax * adxmax + py * py + b.z1 * b.z1;
  u.ok = rmin2 > 1e-6f;  // a point of the box (nearly) at the surface position: no bound
  // 1/rmin, 1/rmax (approximate reciprocal square roots: ~1e-7 relative,
  // far inside the test's margin)
  const float irmin = rsqrtf(fmaxf(rmin2, 1e-6f)), irmax = rsqrtf(fmaxf(rmax2, 1e-6f));
  u.axl = dxl >= 0.0f ? dxl * irmax : dxl * irmin;
  u.axh = dxh >= 0.0f ? dxh * irmin : dxh * irmax;
  u.ayl = py >= 0.0f ? py * irmax : py * irmin;
  u.ayh = py >= 0.0f ? py * irmin : py * irmax;
  u.azl = b.z0 * irmax;
  u.azh = b.z1 * irmin;
  return u;
}
// max of t * v over t in [tlo, thi], v in [vlo, vhi] (a corner of the box)
__device__ __forceinline__ float corner_max(float tlo, float thi, float vlo, float vhi) {
  return fmaxf(fmaxf(tlo * vlo, tlo * vhi), fmaxf(thi * vlo, thi * vhi));
}
__device__ __forceinline__ bool tile_keep(float2 sp, float2 gp, const TileBox &b) {
  const UnitBounds s = unit_bounds(sp.x, sp.y, b), g = unit_bounds(gp.x, gp.y, b);
  if (!s.ok || !g.ok) return true;
  const float uxl = s.axl + g.axl, uxh = s.axh + g.axh;
  const float uyl = s.ayl + g.ayl, uyh = s.ayh + g.ayh;
  const float uzl = s.azl + g.azl, uzh = s.azh + g.azh;
  const float fx1 = uxh + corner_max(-b.t1hi, -b.t1lo, uzl, uzh);
  const float fx2 = corner_max(b.t2lo, b.t2hi, uzl, uzh) - uxl;
  const float fy1 = uyh + corner_max(-b.u1hi, -b.u1lo, uzl, uzh);
  const float fy2 = corner_max(b.u2lo, b.u2hi, uzl, uzh) - uyl;
  const float m = b.margin;
  return !(fx1 < m || fx2 < m || fy1 < m || fy2 < m);  // NaN keeps the member
}

// The surface grid shared by every active point of a tile whose points all
// read the same table cells (one test decides a source's coverage for the
// whole tile).
struct TileGrid {
  float xc, rdx, rdy, hx, hy;
  int nxs, nys;
};
__device__ __forceinline__ bool tile_covers(const TileGrid &g, float2 p) {
  float fx, fy;
  return grid_pos(p.x, p.y, g.xc, g.rdx, g.rdy, g.hx, g.hy, g.nxs, g.nys, fx, fy);
}

template <int NW>
__device__ __forceinline__ float block_min(float v, float (*red)[NW], int k) {
  for (int off = 16; off > 0; off >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = v;
  return v;
}

// Surface weights of a position in a uniform tile's grid: the node offset (in
// table pairs) and the two bilinear weights.  The arithmetic of lookup_tq; the
// position lies on the grid (tile_covers).
__device__ __forceinline__ void surface_weights(const TileGrid &g, float px, float py, int plane,
                                                int &off, float &wx, float &wy) {
  float fx, fy;
  grid_pos(px, py, g.xc, g.rdx, g.rdy, g.hx, g.hy, g.nxs, g.nys, fx, fy);
  const int ix = min((int)fx, max(g.nxs - 2, 0));
  const int iy = min((int)fy, max(g.nys - 2, 0));
  wx = g.nxs > 1 ? __fsub_rn(fx, (float)ix) : 0.0f;
  wy = g.nys > 1 ? __fsub_rn(fy, (float)iy) : 0.0f;
  off = (iy * g.nxs + ix) * plane;
}

// The widened dip limits' ranges over the block's points that take part, in
// rows 0 .. 7 of s_red (8 warps); a barrier later, tile_box reads them.
__device__ __forceinline__ void tile_limits(bool act, float x1c, float x2c, float y1c, float y2c,
                                            float (*s_red)[8]) {
  const float big = 3.0e38f;
  const float v[4] = {x1c, x2c, y1c, y2c};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    block_min<8>(act ? v[j] : big, s_red, 2 * j);
    block_min<8>(act ? -v[j] : big, s_red, 2 * j + 1);
  }
}
__device__ __forceinline__ TileBox tile_box(const float (*s_red)[8], float x0, float x1, float z0,
                                            float z1) {
  float r[8], tmax = 1.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    r[k] = s_red[k][0];
    for (int w = 1; w < 8; ++w) r[k] = fminf(r[k], s_red[k][w]);
    tmax = fmaxf(tmax, fabsf(r[k]));
  }
  TileBox b;
  b.t1lo = r[0], b.t1hi = -r[1], b.t2lo = r[2], b.t2hi = -r[3];
  b.u1lo = r[4], b.u1hi = -r[5], b.u2lo = r[6], b.u2hi = -r[7];
  b.margin = -1e-4f * tmax;
  b.x0 = x0, b.x1 = x1, b.z0 = z0, b.z1 = z1;
  return b;
}

}  // namespace qpsdm
