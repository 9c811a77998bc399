// split_lookup.cuh -- the plain form's field lookups from per-cell records.
//
// The same values as lookup.cuh, bit for bit, with less work: the records
// (fields.h, SplitGrid) hold what bilinear_cell derives from a cell alone,
// and a lane keeps the records of the cell it is in, with the open box of f32
// coordinates that is certain to lie in that cell by the reference's index
// rules of both fields and not on a corner.  A point in the box costs four
// comparisons and the bilinear's own operations; one outside it reads the
// axis cells (two to four 16-byte loads) and, if the cell changed, the
// records (2 + 5 16-byte loads, against 25 scattered loads).  Points on a
// cell's lower edge are resolved there too; every other point (outside the
// grid, on a corner, where f32 rounding and the index rule disagree) takes
// lookup.cuh.
#pragma once

#include "lookup.cuh"
#include "split.cuh"

namespace mr {

// The current's form: a constant, a grid of its own, or a grid whose f32 axes
// equal the bathymetry's (one cell location and one pair of normalised
// coordinates then serve both fields).
enum SplitCurrent : int { SPLIT_CONSTANT = 0, SPLIT_GRID = 1, SPLIT_SAME = 2 };

template <int CUR>
struct SplitCell {
  float xlo = 1.0f, xhi = 0.0f, ylo = 1.0f, yhi = 0.0f;  // the open box (empty)
  int bkey = -1, ckey = -1;       // cells whose records are held
  float bx = 0.0f, by = 0.0f;     // the bathymetry cell's lower axis values
  float cx = 0.0f, cy = 0.0f;     // the current's (SPLIT_GRID)
  float4 h = {}, g = {};          // depth coefficients; dh/dx, dh/dy, m01, m10
  float4 u = {}, v = {}, du = {}, dv = {}, m = {};
};

__device__ __forceinline__ float4 ldg4(const float4 *p) { return __ldg(p); }

// The cell of coordinate t on one axis: true when t is certainly in cell *i,
// strictly inside (*on_edge false) or on its lower axis value.
__device__ __forceinline__ bool axis_cell(const AxisCell *cells, int n, float t, float t0,
                                          float inv, int *i, AxisCell *c, bool *on_edge) {
  // saturating conversion: defined for any t; the cell is checked below
  int k = __float2int_rz((t - t0) * inv);
  k = max(0, min(k, n - 2));
  const float4 a = ldg4(reinterpret_cast<const float4 *>(cells) + k);
  *c = AxisCell{a.x, a.y, a.z, a.w};
  *i = k;
  *on_edge = t == a.w;
  return (t > a.x && t < a.y) || *on_edge;
}

// An empty cell; a constant current is kept in its place from the start.
template <int CUR>
__device__ __forceinline__ void split_start(const CurrentDev &c, SplitCell<CUR> &C) {
  if (CUR == SPLIT_CONSTANT) {
    const F2 u = to_pair(c.cu), v = to_pair(c.cv);
    C.u = make_float4(u.h, u.l, v.h, v.l);
  }
}

// Whether the f64 coordinate v is at or above the threshold of cell i.
__device__ __forceinline__ bool at_or_above(double v, const long long *thr, int i) {
  return order_key_bits(__double_as_longlong(v)) >= __ldg(thr + i);
}

// Moves the lane's records to the cell of (x, y) (f32 tx, ty); false when the
// point needs the general lookup.
template <int CUR>
__device__ __forceinline__ bool split_move(const BathyDev &b, const CurrentDev &c, double x,
                                           double y, float tx, float ty, SplitCell<CUR> &C) {
  int i, j;
  AxisCell xc, yc;
  bool ex, ey;
  const bool inx = axis_cell(b.split.xc, b.split.nx, tx, b.split.x0, b.split.inv_x, &i, &xc, &ex);
  const bool iny = axis_cell(b.split.yc, b.split.ny, ty, b.split.y0, b.split.inv_y, &j, &yc, &ey);
  bool ok = inx && iny && !(ex && ey);
  float xlo = xc.lo, xhi = xc.hi, ylo = yc.lo, yhi = yc.hi;
  int ckey = -1;
  if (CUR != SPLIT_CONSTANT) {
    int ci, cj;
    AxisCell xd, yd;
    bool fx, fy;
    ok &= axis_cell(c.split.xc, c.split.nx, tx, c.split.x0, c.split.inv_x, &ci, &xd, &fx);
    ok &= axis_cell(c.split.yc, c.split.ny, ty, c.split.y0, c.split.inv_y, &cj, &yd, &fy);
    ok &= !(fx && fy);
    if (CUR == SPLIT_SAME) ok &= ci == i && cj == j;
    if (fx) ok &= at_or_above(x, c.xthr, ci);
    if (fy) ok &= at_or_above(y, c.ythr, cj);
    xlo = fmaxf(xlo, xd.lo);
    xhi = fminf(xhi, xd.hi);
    ylo = fmaxf(ylo, yd.lo);
    yhi = fminf(yhi, yd.hi);
    ckey = cj * c.split.nx + ci;
    if (CUR == SPLIT_GRID) {
      C.cx = xd.a1;
      C.cy = yd.a1;
    }
  }
  if (!ok) {
    C.xlo = 1.0f;  // the lower axis values may have moved: an empty box
    C.xhi = 0.0f;
    return false;
  }
  C.xlo = xlo; C.xhi = xhi; C.ylo = ylo; C.yhi = yhi;
  C.bx = xc.a1;
  C.by = yc.a1;
  const int bkey = j * b.split.nx + i;
  if (bkey != C.bkey) {
    const float4 *p = static_cast<const float4 *>(b.split.rec) + static_cast<int64_t>(bkey) * 2;
    C.h = ldg4(p);
    C.g = ldg4(p + 1);
    C.bkey = bkey;
  }
  if (CUR != SPLIT_CONSTANT && ckey != C.ckey) {
    const float4 *p = static_cast<const float4 *>(c.split.rec) + static_cast<int64_t>(ckey) * 5;
    C.u = ldg4(p);
    C.v = ldg4(p + 1);
    C.du = ldg4(p + 2);
    C.dv = ldg4(p + 3);
    if (CUR == SPLIT_GRID) C.m = ldg4(p + 4);
    C.ckey = ckey;
  }
  return true;
}

// cell_apply's operations on coefficients (a00, a10, a01, a11) at normalised
// coordinates (px, py).  Inside a regular cell the inverse's diagonal is
// +-0, so px = m01 tt1 and py = m10 tt0 (adding +-0 changes at most the sign
// of a zero, which the sum below absorbs).
__device__ __forceinline__ float bilinear_record(const float4 &a, float px, float py) {
  return __fadd_rn(__fadd_rn(__fadd_rn(a.x, __fmul_rn(a.y, px)), __fmul_rn(a.z, py)),
                   __fmul_rn(__fmul_rn(a.w, px), py));
}

// The general lookup as a sample; false where the reference has an error.
__device__ __noinline__ static bool split_general(const BathyDev &b, const CurrentDev &c,
                                                  double x, double y, Sample *s) {
  float hg[3];
  double cur[6];
  if (depth_and_gradient<NoCache>(b, d2f(x), d2f(y), hg) != RHS_OK) return false;
  if (current_and_gradient<NoCache>(c, x, y, cur) != RHS_OK) return false;
  s->h = hg[0]; s->gx = hg[1]; s->gy = hg[2];
  s->u = to_pair(cur[0]); s->v = to_pair(cur[1]);
  s->ux = to_pair(cur[2]); s->uy = to_pair(cur[3]);
  s->vx = to_pair(cur[4]); s->vy = to_pair(cur[5]);
  // outside split_ok's domain: NaN depth sends the lane to the FP64 form
  for (float g : {s->gx, s->gy, s->ux.h, s->uy.h, s->vx.h, s->vy.h})
    if (!(fabsf(g) < 1048576.0f)) s->h = f32_nan();
  return true;
}

// The fields at (x, y); false where the reference has an error.
template <int CUR>
__device__ __forceinline__ bool split_sample(const BathyDev &b, const CurrentDev &c, double x,
                                             double y, SplitCell<CUR> &C, Sample &s) {
  const float tx = d2f(x), ty = d2f(y);
  if (!(tx > C.xlo && tx < C.xhi && ty > C.ylo && ty < C.yhi)) {
    if (!split_move<CUR>(b, c, x, y, tx, ty, C)) {
      Sample t;  // its address escapes; s stays in registers
      if (!split_general(b, c, x, y, &t)) return false;
      s = t;
      return true;
    }
  }
  const float px = __fmul_rn(C.g.z, __fsub_rn(ty, C.by));  // :74
  const float py = __fmul_rn(C.g.w, __fsub_rn(tx, C.bx));  // :75
  s.h = bilinear_record(C.h, px, py);
  s.gx = C.g.x;
  s.gy = C.g.y;
  if (CUR == SPLIT_CONSTANT) {
    s.u = F2{C.u.x, C.u.y};  // set once by split_start
    s.v = F2{C.u.z, C.u.w};
    s.ux = s.uy = s.vx = s.vy = F2{0.0f, 0.0f};
  } else {
    float qx = px, qy = py;
    if (CUR == SPLIT_GRID) {
      qx = __fmul_rn(C.m.x, __fsub_rn(ty, C.cy));
      qy = __fmul_rn(C.m.y, __fsub_rn(tx, C.cx));
    }
    s.u = F2{bilinear_record(C.u, qx, qy), 0.0f};
    s.v = F2{bilinear_record(C.v, qx, qy), 0.0f};
    s.ux = F2{C.du.x, C.du.y};
    s.uy = F2{C.du.z, C.du.w};
    s.vx = F2{C.dv.x, C.dv.y};
    s.vy = F2{C.dv.z, C.dv.w};
  }
  return true;
}

}  // namespace mr
