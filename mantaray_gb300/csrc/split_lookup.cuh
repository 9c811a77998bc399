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
// equal the bathymetry's (both fields then share m01 and m10).
enum SplitCurrent : int { SPLIT_CONSTANT = 0, SPLIT_GRID = 1, SPLIT_SAME = 2 };

template <int CUR>
struct SplitCell {
  float xlo = 1.0f, xhi = 0.0f, ylo = 1.0f, yhi = 0.0f;  // the open box (empty)
  int bkey = -1, ckey = -1;       // cells whose records are held
  float bx = 0.0f, by = 0.0f;     // the bathymetry cell's lower axis values
  float cx = 0.0f, cy = 0.0f;     // the current cell's
  float4 h = {}, g = {};          // depth coefficients; dh/dx, dh/dy, m01, m10
  float4 u = {}, v = {};          // (u00, v00, u10, v10), (u01, v01, u11, v11)
  float4 du = {}, dv = {};        // (d/dx, d/dy) high halves, then low
  float4 m = {};                  // m01, m10 (SPLIT_GRID)
};

__device__ __forceinline__ float4 ldg4(const float4 *p) { return __ldg(p); }

// The cell of coordinate t on one axis: true when t is certainly in cell *i,
// strictly inside (*on_edge false) or on its lower axis value.
__device__ __forceinline__ bool axis_cell(const AxisCell *cells, int n, float t, float t0,
                                          float inv, float sp, int uniform, int *i, AxisCell *c,
                                          bool *on_edge) {
  // saturating conversion: defined for any t; the cell is checked below
  int k = __float2int_rz((t - t0) * inv);
  k = max(0, min(k, n - 2));
  if (uniform) {
    const float f = static_cast<float>(k);
    c->lo = c->a1 = c->edge = __fmaf_rn(f, sp, t0);
    c->hi = __fmaf_rn(f + 1.0f, sp, t0);
  } else {
    const float4 a = ldg4(reinterpret_cast<const float4 *>(cells) + k);
    *c = AxisCell{a.x, a.y, a.z, a.w};
  }
  *i = k;
  *on_edge = t == c->edge;
  return (t > c->lo && t < c->hi) || *on_edge;
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

// Moves the lane's records to the cell of (tx, ty); false when the point
// needs the general lookup.  at() gives its f64 coordinates.  A point whose
// f32 coordinate is on a cell's lower axis value is in that cell for the
// bathymetry (its rule is on the f32 coordinate) and in that cell or the one
// below for the current (its rule is on the f64 coordinate): rays along a
// grid line stay there for many steps.
template <int CUR, typename At>
__device__ __forceinline__ bool split_move(const BathyDev &b, const CurrentDev &c, float tx,
                                           float ty, At at, SplitCell<CUR> &C) {
  int i, j;
  AxisCell xc, yc;
  bool ex, ey;
  const SplitGrid &g = b.split;
  const bool inx = axis_cell(g.xc, g.nx, tx, g.x0, g.inv_x, g.sp_x, g.uniform_x, &i, &xc, &ex);
  const bool iny = axis_cell(g.yc, g.ny, ty, g.y0, g.inv_y, g.sp_y, g.uniform_y, &j, &yc, &ey);
  bool ok = inx && iny && !(ex && ey);
  bool below = false;
  float xlo = xc.lo, xhi = xc.hi, ylo = yc.lo, yhi = yc.hi;
  int ckey = -1;
  if (CUR != SPLIT_CONSTANT) {
    int ci, cj;
    AxisCell xd, yd;
    bool fx, fy;
    const SplitGrid &d = c.split;
    ok &= axis_cell(d.xc, d.nx, tx, d.x0, d.inv_x, d.sp_x, d.uniform_x, &ci, &xd, &fx);
    ok &= axis_cell(d.yc, d.ny, ty, d.y0, d.inv_y, d.sp_y, d.uniform_y, &cj, &yd, &fy);
    ok &= !(fx && fy);
    if (CUR == SPLIT_SAME) ok &= ci == i && cj == j;
    xlo = fmaxf(xlo, xd.lo);
    xhi = fminf(xhi, xd.hi);
    ylo = fmaxf(ylo, yd.lo);
    yhi = fminf(yhi, yd.hi);
    C.cx = xd.a1;
    C.cy = yd.a1;
    if (ok && (fx || fy)) {
      double x, y;
      at(&x, &y);
      below = fx ? !at_or_above(x, c.xthr, ci) : !at_or_above(y, c.ythr, cj);
      if (below) {
        ci -= fx;
        cj -= fy;
        ok = ci >= 0 && cj >= 0;
        if (ok && fx) C.cx = __ldg(&d.xc[ci].a1);
        if (ok && fy) C.cy = __ldg(&d.yc[cj].a1);
      }
    }
    ckey = cj * c.split.nx + ci;
  }
  // no box where the fields' cells differ, or where the records do not apply
  // (the lower axis values have moved)
  C.xlo = ok && !below ? xlo : 1.0f;
  C.xhi = ok && !below ? xhi : 0.0f;
  C.ylo = ylo;
  C.yhi = yhi;
  if (!ok) return false;
  C.bx = xc.a1;
  C.by = yc.a1;
  const int bkey = j * b.split.nx + i;
  if (bkey != C.bkey) {
    const float4 *p = static_cast<const float4 *>(b.split.rec) + static_cast<int64_t>(bkey) * 2;
    C.h = ldg4(p);
    C.g = ldg4(p + 1);
    C.bkey = bkey;
  }
  if (CUR != SPLIT_CONSTANT) {
    const float4 *p = static_cast<const float4 *>(c.split.rec) + static_cast<int64_t>(ckey) * 5;
    if (ckey != C.ckey) {
      C.u = ldg4(p);
      C.v = ldg4(p + 1);
      C.du = ldg4(p + 2);
      C.dv = ldg4(p + 3);
      if (CUR == SPLIT_GRID) C.m = ldg4(p + 4);
      C.ckey = ckey;
    }
    if (CUR == SPLIT_SAME && below) {  // the cell below may be of another size
      const float4 m = ldg4(p + 4);
      return m.x == C.g.z && m.y == C.g.w;
    }
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
// The same for u and v at once: coefficients (u00, v00, u10, v10) and (u01,
// v01, u11, v11).  The products are packed, the sums scalar: ptxas contracts
// a packed product and sum into one FMA, whatever -fmad and the rounding
// modifiers say, which would change the reference's rounding.
__device__ __forceinline__ V bilinear_record2(const float4 &a, const float4 &b, float px,
                                              float py) {
  const V p = vmul(V{a.z, a.w}, both(px)), q = vmul(V{b.x, b.y}, both(py)),
          r = vmul(vmul(V{b.z, b.w}, both(px)), both(py));
  return V{__fadd_rn(__fadd_rn(__fadd_rn(a.x, p.x), q.x), r.x),
           __fadd_rn(__fadd_rn(__fadd_rn(a.y, p.y), q.y), r.y)};
}

// The general lookup as a sample; false where the reference has an error.
__device__ __noinline__ static bool split_general(const BathyDev &b, const CurrentDev &c,
                                                  double x, double y, Sample *s) {
  float hg[3];
  double cur[6];
  if (depth_and_gradient<NoCache>(b, d2f(x), d2f(y), hg) != RHS_OK) return false;
  if (current_and_gradient<NoCache>(c, x, y, cur) != RHS_OK) return false;
  F2 p[6];
  for (int q = 0; q < 6; ++q) p[q] = to_pair(cur[q]);
  s->h = hg[0];
  s->g = V{hg[1], hg[2]};
  s->uv = V2{V{p[0].h, p[1].h}, V{p[0].l, p[1].l}};
  s->du = V2{V{p[2].h, p[3].h}, V{p[2].l, p[3].l}};
  s->dv = V2{V{p[4].h, p[5].h}, V{p[4].l, p[5].l}};
  // outside split_ok's domain: NaN depth sends the lane to the FP64 form
  for (float g : {hg[1], hg[2], p[2].h, p[3].h, p[4].h, p[5].h})
    if (!(fabsf(g) < 1048576.0f)) s->h = f32_nan();
  return true;
}

// The fields at the f64 point whose f32 coordinates are (tx, ty); at() gives
// its f64 coordinates, needed only off the fast path.  False where the
// reference has an error.
template <int CUR, typename At>
__device__ __forceinline__ bool split_sample(const BathyDev &b, const CurrentDev &c, float tx,
                                             float ty, At at, SplitCell<CUR> &C, Sample &s) {
  if (!(tx > C.xlo && tx < C.xhi && ty > C.ylo && ty < C.yhi)) {
    if (!split_move<CUR>(b, c, tx, ty, at, C)) {
      double x, y;
      at(&x, &y);
      Sample t;  // its address escapes; s stays in registers
      if (!split_general(b, c, x, y, &t)) return false;
      s = t;
      return true;
    }
  }
  const V p = vmul(V{C.g.z, C.g.w}, vsub(V{ty, tx}, V{C.by, C.bx}));  // :74, :75
  s.h = bilinear_record(C.h, p.x, p.y);
  s.g = V{C.g.x, C.g.y};
  if (CUR == SPLIT_CONSTANT) {  // set once by split_start
    s.uv = V2{V{C.u.x, C.u.z}, V{C.u.y, C.u.w}};
    s.du = s.dv = zero2();
  } else {
    const V m = CUR == SPLIT_GRID ? V{C.m.x, C.m.y} : V{C.g.z, C.g.w};
    const V q = vmul(m, vsub(V{ty, tx}, V{C.cy, C.cx}));
    s.uv = V2{bilinear_record2(C.u, C.v, q.x, q.y), both(0.0f)};
    s.du = V2{V{C.du.x, C.du.y}, V{C.du.z, C.du.w}};
    s.dv = V2{V{C.dv.x, C.dv.y}, V{C.dv.z, C.dv.w}};
  }
  return true;
}

}  // namespace mr
