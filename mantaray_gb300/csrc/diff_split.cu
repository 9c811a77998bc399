// diff_split.cu -- the FP64 differentiation form (forward with checkpoints,
// adjoint, tangent-linear; model and derivations in diff.cu) on float pairs.
//
// GB300's FP64 pipe issues 2 lanes per SM and clock and takes 64 cycles an
// operation, so the FP64 kernels of diff.cu keep it 70% busy with 8% of the
// issue slots used.  Here the stages run on pairs of floats (split.cuh), with
// one FP64 anchor a step for each quantity whose error would otherwise add up
// along the ray:
//   the state:     as x, y in split.cuh: the first stage's derivative in FP64,
//                  the stages' differences from it in pairs;
//   d(x)/d(k):     M = d(c_g k/|k|)/dk, the term by which a wavenumber tangent
//                  (position adjoint) feeds the position tangent (wavenumber
//                  adjoint) at every step, in FP64 at one state of the step,
//                  the stages' differences from it in pairs;
//   all the rest   (refraction and current terms of the tangent and adjoint) is
//                  a small part per step of what it is added to in FP64, and is
//                  taken from the pairs, with the product of the low halves
//                  kept (MR_SPLIT_LOW_PRODUCT: 7% of the time; without it the
//                  gradients' error after 300 steps is 1.7 times FP64's).
//
// 32,768 rays x 300 steps on 512 x 512 nodes, forward and adjoint: 44.0 ms in
// FP64, 14.1 ms here (0.6 less with the wavenumbers' derivative in pairs alone,
// whose error under strong refraction, depths 200 times apart in neighbouring
// cells, was 6 times FP64's).  The recomputed forward pass and the adjoint are
// 2,800 and 7,300 instructions a warp-step, two warps a scheduler: what is left
// is the latency of dependent FP32 operations (2.3 of 4.6 cycles an
// instruction), and the lanes of a warp in deep and in shallower water (22.5 of
// 32 active).  The variant with FP64 equations in the reverse pass took 17.8 ms.
// Tangent-linear, 8,192 rays x 500 steps: 16.2 ms in FP64, 5.7 here, one warp a
// scheduler (5.3 with one unit for the call, which lost the tangents of every
// ray far below the call's largest); along a depth tangent alone 5.8 (29.6:
// lanes parted by steps in FP64 stayed parted).
// Error against 128-bit arithmetic over 50 to 400 steps of 1 to 4 s on 200 to
// 600 nodes a side, norm over norm, as a fraction of the FP64 kernels' error
// (geometric mean of 8 cases): end positions and wavenumbers 0.97, gradients
// by initial position 0.56, wavenumber 0.74, depth 0.82, u 1.06 (2.4e-15 at
// 50 steps), v 0.96; tangents of position 0.75, of wavenumber 0.82.
//
// With a = kh, N = 2a / sinh 2a, C = 2a coth 2a, I = 1 / sinh 2a and sigma =
// sqrt(g k tanh a) (identities of the definitions):
//   w = c_g / k = sigma (1 + N) / (2 k^2)       f = -k sigma I
//   c_g,k = sigma / (2 k^2) ((N^2 - 1)/2 + N (1 - C))
//   c_g,h = -f,k = sigma I (3/2 + N/2 - C)
//   f,h = sigma k^2 I (2 (1 + E^2)/(1 - E^2) - I),  E = exp(-2a)
// and, beyond a = 22, w = sqrt(g)/2 k^(-3/2), c_g,k = -w/2, the rest 0.
//
// Fields: one record per cell, built at the start of the call (bilinear
// coefficients of depth, u and v in pairs and in FP64, 192 bytes; of the
// tangent fields in pairs, 108), kept in registers while a ray stays in the
// cell.  A stage's position is the step's
// FP64 cell and fraction plus the displacement in pairs.
//
// Steps outside the pairs' domain (depth or k^2 as in split_ok, a cell
// outside the grid, the grid's closed far edge) run the FP64 functions of
// diff.cuh.  Compiled with -fmad=false.

#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>
#include <vector>

#define MR_SPLIT_LOW_PRODUCT
#include "diff.cuh"
#include "diff_split.h"
#include "split.cuh"

namespace mr {

namespace {

constexpr int kSplitBlock = 64;
constexpr double kHalfSqrtG = 0x1.90b410d07f01ep+0;  // sqrt(9.8) / 2

// One grid as the kernels read it: its axes, and per cell (by j (nx - 1) + i)
// the pair records and the FP64 ones.  Bathymetry: 2 float4 (c0 cx cy cxy:
// high halves, low halves) and 2 double2; current: 4 float4 ((u v) of c0 and
// cx, of cy and cxy: high, then low) and 4 double2 ((u v) of c0, cx, cy, cxy).
struct SplitField {
  const float4 *rec;
  const double2 *rec64;
  int nx, ny;
  double x0, y0, inv_dx, inv_dy;
  V2 inv;  // (1/dx, 1/dy) as pairs
};

struct SplitArgs {
  DiffArgs<double> A;
  SplitField b, c;
  double sixth;
  F2 dt2, half2, sixth2;
};

// Cell `cell`'s bilinear coefficients of nodes a.
__device__ __forceinline__ void coefficients(const double *a, int nx, int64_t cell, double o[4]) {
  const int64_t base = cell / (nx - 1) * nx + cell % (nx - 1);
  const double v00 = a[base], v10 = a[base + 1], v01 = a[base + nx], v11 = a[base + nx + 1];
  o[0] = v00;
  o[1] = v10 - v00;
  o[2] = v01 - v00;
  o[3] = ((v11 - v10) - v01) + v00;
}

// A bathymetry's (current's) cell as pairs and in FP64.
__device__ __forceinline__ void bathy_record(const double *a, int nx, int64_t k, float4 *b,
                                             double2 *b64) {
  double o[4];
  coefficients(a, nx, k, o);
  F2 q[4];
  for (int t = 0; t < 4; ++t) q[t] = to_pair(o[t]);
  b[2 * k] = make_float4(q[0].h, q[1].h, q[2].h, q[3].h);
  b[2 * k + 1] = make_float4(q[0].l, q[1].l, q[2].l, q[3].l);
  b64[2 * k] = make_double2(o[0], o[1]);
  b64[2 * k + 1] = make_double2(o[2], o[3]);
}
__device__ __forceinline__ void current_record(const double *u, const double *v, int nx, int64_t k,
                                               float4 *c, double2 *c64) {
  double o[4], p[4];
  coefficients(u, nx, k, o);
  coefficients(v, nx, k, p);
  F2 q[4], r[4];
  for (int t = 0; t < 4; ++t) {
    q[t] = to_pair(o[t]);
    r[t] = to_pair(p[t]);
    c64[4 * k + t] = make_double2(o[t], p[t]);
  }
  c[4 * k] = make_float4(q[0].h, r[0].h, q[1].h, r[1].h);
  c[4 * k + 1] = make_float4(q[2].h, r[2].h, q[3].h, r[3].h);
  c[4 * k + 2] = make_float4(q[0].l, r[0].l, q[1].l, r[1].l);
  c[4 * k + 3] = make_float4(q[2].l, r[2].l, q[3].l, r[3].l);
}

__global__ void build_diff_records(SplitArgs S, float4 *b, double2 *b64, float4 *c, double2 *c64) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < static_cast<int64_t>(S.b.nx - 1) * (S.b.ny - 1))
    bathy_record(S.A.bg.a, S.b.nx, k, b, b64);
  if (k < static_cast<int64_t>(S.c.nx - 1) * (S.c.ny - 1))
    current_record(S.A.cg.a, S.A.cg.b, S.c.nx, k, c, c64);
}

// The cells a lane holds.
struct DiffCell {
  int bkey = -1, ckey = -1;
  float4 b[2], c[4];
  __device__ __forceinline__ F2 h0() const { return F2{b[0].x, b[1].x}; }
  __device__ __forceinline__ F2 hx() const { return F2{b[0].y, b[1].y}; }
  __device__ __forceinline__ F2 hy() const { return F2{b[0].z, b[1].z}; }
  __device__ __forceinline__ F2 hxy() const { return F2{b[0].w, b[1].w}; }
  // (u, v) lanes
  __device__ __forceinline__ V2 w0() const { return V2{V{c[0].x, c[0].y}, V{c[2].x, c[2].y}}; }
  __device__ __forceinline__ V2 wx() const { return V2{V{c[0].z, c[0].w}, V{c[2].z, c[2].w}}; }
  __device__ __forceinline__ V2 wy() const { return V2{V{c[1].x, c[1].y}, V{c[3].x, c[3].y}}; }
  __device__ __forceinline__ V2 wxy() const { return V2{V{c[1].z, c[1].w}, V{c[3].z, c[3].w}}; }
};

// A step's first point on one grid: cell and fractions in FP64.
struct Base {
  int i, j;
  V2 f;          // fractions as pairs
  double fx, fy;
};

// False when the point is outside (or on the closed far edge, or NaN).
__device__ __forceinline__ bool base_of(const SplitField &g, double x, double y, Base *b) {
  const double ix = (x - g.x0) * g.inv_dx, iy = (y - g.y0) * g.inv_dy;
  // floor: the f32 guess is off by one at most, and corrected
  float gi = floorf(d2f(ix)), gj = floorf(d2f(iy));
  if (!(gi >= -1.0f && gi <= static_cast<float>(g.nx) && gj >= -1.0f &&
        gj <= static_cast<float>(g.ny)))
    return false;
  double fx = ix - f2d_zero(gi), fy = iy - f2d_zero(gj);
  if (bits_of(fx) >> 63 && fx != 0.0) { fx += 1.0; gi -= 1.0f; }
  if (bits_of(fy) >> 63 && fy != 0.0) { fy += 1.0; gj -= 1.0f; }
  b->i = static_cast<int>(gi);
  b->j = static_cast<int>(gj);
  b->fx = fx;
  b->fy = fy;
  const F2 px = to_pair(fx), py = to_pair(fy);
  b->f = V2{V{px.h, py.h}, V{px.l, py.l}};
  return b->i >= 0 && b->i <= g.nx - 2 && b->j >= 0 && b->j <= g.ny - 2;
}

// The cell and fractions of a point displaced from the base by d (pairs).
__device__ __forceinline__ bool displaced(const SplitField &g, const Base &b, V2 d, int *i, int *j,
                                          V2 *f) {
  const V2 u = add(b.f, mul(d, g.inv));
  const V s = vadd(u.h, u.l);
  V l = vsub(u.l, vsub(s, u.h));
  V fl = V{floorf(s.x), floorf(s.y)};
  // a low half below zero at an integer: the cell below
  if (s.x == fl.x && l.x < 0.0f) fl.x -= 1.0f;
  if (s.y == fl.y && l.y < 0.0f) fl.y -= 1.0f;
  // s - fl exactly: -0.05 + 1 does not fit the high half
  const V hi = vsub(s, fl);
  *f = V2{hi, vadd(l, vsub(s, vadd(hi, fl)))};
  *i = b.i + __float2int_rz(fl.x);  // saturates; bounded by the test below
  *j = b.j + __float2int_rz(fl.y);
  return fabsf(fl.x) < 1048576.0f && fabsf(fl.y) < 1048576.0f && *i >= 0 && *i <= g.nx - 2 &&
         *j >= 0 && *j <= g.ny - 2;
}

// The fields at a point, in pairs, with what the partials need.
struct At {
  V2 fb, fc;    // fractions on the two grids
  F2 h, hx, hy; // depth; its bilinear surface's derivatives per cell
  V2 uv, wx, wy;  // (u, v) and theirs
};

__device__ __forceinline__ float4 ld4(const float4 *p) { return __ldg(p); }

template <bool SAME>
__device__ __forceinline__ void take_cells(const SplitArgs &S, int bi, int bj, int ci, int cj,
                                           DiffCell &C) {
  const int bkey = bj * (S.b.nx - 1) + bi;
  if (bkey != C.bkey) {
    const float4 *p = S.b.rec + static_cast<int64_t>(bkey) * 2;
    C.b[0] = ld4(p);
    C.b[1] = ld4(p + 1);
    C.bkey = bkey;
  }
  const int ckey = SAME ? bkey : cj * (S.c.nx - 1) + ci;
  if (ckey != C.ckey) {
    const float4 *p = S.c.rec + static_cast<int64_t>(ckey) * 4;
#pragma unroll
    for (int q = 0; q < 4; ++q) C.c[q] = ld4(p + q);
    C.ckey = ckey;
  }
}

template <bool SAME>
__device__ __forceinline__ void fields_at(const DiffCell &C, V2 fb, V2 fc, At *p) {
  p->fb = fb;
  p->fc = SAME ? fb : fc;
  const F2 fx = x_of(fb), fy = y_of(fb);
  p->hx = add(C.hx(), mul(C.hxy(), fy));
  p->hy = add(C.hy(), mul(C.hxy(), fx));
  p->h = add(add(C.h0(), mul(C.hx(), fx)), mul(p->hy, fy));
  const V2 gx = both(x_of(p->fc)), gy = both(y_of(p->fc));
  p->wx = add(C.wx(), mul(C.wxy(), gy));
  p->wy = add(C.wy(), mul(C.wxy(), gx));
  p->uv = add(add(C.w0(), mul(C.wx(), gx)), mul(p->wy, gy));
}

__device__ __forceinline__ bool diff_ok(const At &p, float k2) {
  return p.h.h > 0.0078125f && p.h.h < 131072.0f && fabsf(p.uv.h.x) < 1048576.0f &&
         fabsf(p.uv.h.y) < 1048576.0f && fabsf(p.hx.h) < 1048576.0f &&
         fabsf(p.hy.h) < 1048576.0f && k2 > 0x1p-40f && k2 < 0x1p20f;
}

// What the equations need at a state: w = c_g / k and f, and with PARTIALS
// c_g,k, c_g,h and f,h (zero in deep water, as f).  anchor: also w in FP64 at
// (kx, ky) and depth hd, and with PARTIALS beta = (c_g,k - w) / k^2 (M = w I +
// beta k k^T), from the pairs' quantities with one Newton correction each.
struct Eqs { F2 w, f, qk, qh, fh; };

template <bool PARTIALS>
__device__ __forceinline__ void eqs_of(const Wave &wv, F2 h, Eqs *e, bool anchor, double kx,
                                       double ky, double hd, double *w64, double *beta64,
                                       double *f64 = nullptr) {
  const F2 kC2 = F2{0x1.90b41p+1f, 0x1.a0fe04p-24f};  // sqrt(9.8)
  const F2 a = mul(wv.k, h);
  if (a.h > 22.0f) {
    const F2 w0 = mul(wv.rk, rsqrt2(wv.k));
    e->w = mul(scale(0.5f, kC2), w0);
    e->f = F2{0.0f, 0.0f};
    if (PARTIALS) {
      e->qk = scale(-0.5f, e->w);
      e->qh = e->fh = e->f;
    }
    if (anchor) {
      const double k2d = fma(kx, kx, ky * ky);
      const double wd = to_double(w0);
      const double w2 = wd * wd;
      const double c = fma(-quarter_of(w2 * w2), k2d * k2d * k2d, 0.25);
      *w64 = kHalfSqrtG * fma(wd, c, wd);
      if (f64) *f64 = 0.0;
      if (PARTIALS) {
        const double r0 = to_double(wv.rk);
        const double r2 = r0 * r0;  // 1/k^2 to 2^-45: one correction
        *beta64 = -1.5 * *w64 * fma(r2, fma(-k2d, r2, 1.0), r2);
      }
    }
    return;
  }
  int n;
  F2 E, m;
  const F2 an = fast_two_sum(a.h, a.l);
  split_exp(scale(-2.0f, an), &n, &E, &m);
  const F2 one = fast_two_sum(1.0f, E.h);
  const F2 p1 = F2{one.h, one.l + E.l};
  const F2 rho = rsqrt2(mul(mul(wv.k, m), p1));   // 1 / sqrt(k (1 - E^2))
  const F2 kR = mul(wv.k, sqr(rho));              // 1 / (1 - E^2)
  const F2 I = scale(2.0f, mul(E, kR));
  const F2 N = scale(2.0f, mul(a, I));
  const F2 sg = mul(kC2, mul(mul(wv.k, m), rho)); // sigma
  const F2 one_n = add_f(N, 1.0f);
  const F2 rk2 = sqr(wv.rk);
  const F2 s2 = scale(0.5f, mul(sg, rk2));        // sigma / (2 k^2)
  e->w = mul(s2, one_n);
  const F2 sI = mul(sg, I);
  e->f = neg(mul(wv.k, sI));
  if (PARTIALS) {
    const F2 coth = mul(add_f(sqr(E), 1.0f), kR);
    const F2 C = scale(2.0f, mul(a, coth));
    const F2 one_c = add_f(neg(C), 1.0f);
    e->qk = mul(s2, add(scale(0.5f, add_f(sqr(N), -1.0f)), mul(N, one_c)));
    e->qh = mul(sI, add(scale(0.5f, one_n), one_c));
    e->fh = mul(mul(sI, wv.k2), add(scale(2.0f, coth), neg(I)));
  }
  if (anchor) {
    const double k2d = fma(kx, kx, ky * ky);
    const double rk0 = to_double(wv.rk);
    const double k0 = k2d * rk0;
    const double ek = fma(-half_of(k0), rk0, 0.5);
    const double kd = fma(k0, ek, k0);
    const double rkd = fma(rk0, ek, rk0);
    const double ad = kd * hd;
    double Ed, md;
    anchor_exp(ad, n, &Ed, &md);
    const double km = kd * md;
    const double D = km * (1.0 + Ed);
    const double r0 = to_double(rho);
    const double er = fma(-half_of(D * r0), r0, 0.5);
    const double rhod = fma(r0, er, r0);
    const double kRd = kd * (rhod * rhod);
    const double Nd = 4.0 * ad * (Ed * kRd);
    const double rk2d = rkd * rkd;
    const double sgd = kHalfSqrtG * (km * rhod);   // sigma / 2
    const double s2d = sgd * rk2d;
    if (f64) *f64 = -4.0 * (kd * sgd) * (Ed * kRd);
    *w64 = fma(s2d, Nd, s2d);
    if (PARTIALS) {
      const double one_cd = fma(-2.0 * ad, fma(Ed, Ed, 1.0) * kRd, 1.0);
      const double qkd = s2d * fma(Nd, one_cd, fma(0.5 * Nd, Nd, -0.5));
      *beta64 = (qkd - *w64) * rk2d;
    }
  }
}

__device__ __forceinline__ F2 sum_lanes(V2 a) { return add(x_of(a), y_of(a)); }

// (dx, dy) and (dkx, dky).
__device__ __forceinline__ void derivative(const SplitArgs &S, const DiffCell &C, const Wave &wv,
                                           const At &p, const Eqs &e, V2 *d, V2 *dk) {
  *d = add(mul(both(e.w), wv.kv), p.uv);
  const F2 tx = sum_lanes(mul(wv.kv, C.wx())), ty = sum_lanes(mul(wv.kv, C.wy()));
  const V2 t = mul(V2{V{tx.h, ty.h}, V{tx.l, ty.l}}, S.c.inv);
  const V2 g = V2{V{C.b[0].y, C.b[0].z}, V{C.b[1].y, C.b[1].z}};
  *dk = sub(mul(mul(both(e.f), g), S.b.inv), t);
}

__device__ __forceinline__ V2 lanes(F2 a, F2 b) { return V2{V{a.h, b.h}, V{a.l, b.l}}; }

// FP64 fields at the base point: depth, and all of them.
__device__ __forceinline__ double depth64(const SplitArgs &S, const Base &b) {
  const double2 *p = S.b.rec64 + static_cast<int64_t>(b.j * (S.b.nx - 1) + b.i) * 2;
  const double2 p0 = __ldg(p), p1 = __ldg(p + 1);
  return fma(b.fy, fma(b.fx, p1.y, p1.x), fma(b.fx, p0.y, p0.x));
}
struct Fields64 {
  double h, u, v;            // at the point
  double gx, gy;             // depth's cell gradient
  double ux, uy, vx, vy;     // (u, v)'s
};
template <bool SAME>
__device__ __forceinline__ Fields64 fields64(const SplitArgs &S, const Base &b, const Base &c) {
  const double2 *p = S.b.rec64 + static_cast<int64_t>(b.j * (S.b.nx - 1) + b.i) * 2;
  const double2 p0 = __ldg(p), p1 = __ldg(p + 1);
  const Base &g = SAME ? b : c;
  const double2 *q = S.c.rec64 + static_cast<int64_t>(g.j * (S.c.nx - 1) + g.i) * 4;
  const double2 q0 = __ldg(q), q1 = __ldg(q + 1), q2 = __ldg(q + 2), q3 = __ldg(q + 3);
  Fields64 f;
  f.h = fma(b.fy, fma(b.fx, p1.y, p1.x), fma(b.fx, p0.y, p0.x));
  f.u = fma(g.fy, fma(g.fx, q3.x, q2.x), fma(g.fx, q1.x, q0.x));
  f.v = fma(g.fy, fma(g.fx, q3.y, q2.y), fma(g.fx, q1.y, q0.y));
  f.gx = p0.y * S.b.inv_dx;
  f.gy = p1.x * S.b.inv_dy;
  f.ux = q1.x * S.c.inv_dx;
  f.vx = q1.y * S.c.inv_dx;
  f.uy = q2.x * S.c.inv_dy;
  f.vy = q2.y * S.c.inv_dy;
  return f;
}

// The right-hand side at the base point in FP64.
__device__ __forceinline__ void anchors(const Fields64 &F, const double y[4], double w, double f,
                                        double a[4]) {
  a[0] = fma(w, y[2], F.u);
  a[1] = fma(w, y[3], F.v);
  a[2] = fma(f, F.gx, -fma(y[2], F.ux, y[3] * F.vx));
  a[3] = fma(f, F.gy, -fma(y[2], F.uy, y[3] * F.vy));
}

// The stage point at displacement disp and wavenumber kv; false outside.
template <bool SAME>
__device__ __forceinline__ bool stage_at(const SplitArgs &S, const Base &b, const Base &c, V2 disp,
                                         DiffCell &C, At *p) {
  int bi, bj, ci = 0, cj = 0;
  V2 fb, fc = zero2();
  bool ok = displaced(S.b, b, disp, &bi, &bj, &fb);
  if (!SAME) ok &= displaced(S.c, c, disp, &ci, &cj, &fc);
  if (!ok) return false;
  take_cells<SAME>(S, bi, bj, ci, cj, C);
  fields_at<SAME>(C, fb, fc, p);
  return true;
}

// The stages of a step from y: displacements and wavenumbers of stages 2-4
// (disp[q], kq[q]) where STORE, and the new state in yn.  False when a stage
// is outside the pairs' domain.
template <bool SAME, typename Store>
__device__ __forceinline__ bool forward_step(const SplitArgs &S, DiffCell &C, const double y[4],
                                             double yn[4], Store store) {
  Base b, c;
  if (!base_of(S.b, y[0], y[1], &b)) return false;
  if (!SAME && !base_of(S.c, y[0], y[1], &c)) return false;
  take_cells<SAME>(S, b.i, b.j, SAME ? 0 : c.i, SAME ? 0 : c.j, C);
  At p;
  fields_at<SAME>(C, b.f, SAME ? b.f : c.f, &p);
  const V2 k = lanes(to_pair(y[2]), to_pair(y[3]));
  Wave wv = wave_of(k);
  bool ok = diff_ok(p, wv.k2.h);
  double w64, f64;
  Eqs e;
  V2 d1, d, dk;
  double a[4];
  {
    const Fields64 F = fields64<SAME>(S, b, c);
    eqs_of<false>(wv, p.h, &e, true, y[2], y[3], F.h, &w64, nullptr, &f64);
    anchors(F, y, w64, f64, a);
  }
  derivative(S, C, wv, p, e, &d1, &dk);
  const V2 k1 = dk;
  V2 sd = zero2(), sk = sd;
  d = d1;
#pragma unroll 1
  for (int st = 0; st < 3; ++st) {
    if (!ok) return false;
    const V2 hs = both(st == 2 ? S.dt2 : S.half2);
    const V2 disp = mul(d, hs), q = add(k, mul(dk, hs));
    store(st, disp, q);
    wv = wave_of(q);
    if (!stage_at<SAME>(S, b, c, disp, C, &p)) return false;
    ok = diff_ok(p, wv.k2.h);
    eqs_of<false>(wv, p.h, &e, false, 0.0, 0.0, 0.0, nullptr, nullptr);
    derivative(S, C, wv, p, e, &d, &dk);
    const float wt = st == 2 ? 1.0f : 2.0f;
    sd = add(sd, scale(wt, sub(d, d1)));
    sk = add(sk, scale(wt, sub(dk, k1)));
  }
  if (!ok) return false;
  const V2 s6 = mul(sd, both(S.sixth2)), k6 = mul(sk, both(S.sixth2));
  yn[0] = y[0] + (fma(S.A.dt, a[0], f2d_zero(s6.h.x)) + f2d_zero(s6.l.x));
  yn[1] = y[1] + (fma(S.A.dt, a[1], f2d_zero(s6.h.y)) + f2d_zero(s6.l.y));
  yn[2] = y[2] + (fma(S.A.dt, a[2], f2d_zero(k6.h.x)) + f2d_zero(k6.l.x));
  yn[3] = y[3] + (fma(S.A.dt, a[3], f2d_zero(k6.h.y)) + f2d_zero(k6.l.y));
  return true;
}

__device__ __noinline__ bool fp64_rk4(const DiffArgs<double> &A, double *y) {
  double s[4] = {y[0], y[1], y[2], y[3]};
  Held<double> N;
  if (!rk4(A, s, N)) return false;
#pragma unroll
  for (int q = 0; q < 4; ++q) y[q] = s[q];
  return true;
}

template <bool SAME>
__global__ void __launch_bounds__(kSplitBlock, 6)
    diff_split_forward(const __grid_constant__ SplitArgs S) {
  const DiffArgs<double> &A = S.A;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  double y[4] = {A.x0[i], A.y0[i], A.kx0[i], A.ky0[i]};
  bool ok = true;
  DiffCell C;
  int64_t to_ck = 0;
  double *ck = A.ckpt + i;
  for (int64_t s = 0; s < A.steps; ++s) {
    if (to_ck == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) ck[q * A.n] = y[q];
      ck += 4 * A.n;
      to_ck = A.ck_every;
    }
    --to_ck;
    double yn[4];
    if (!forward_step<SAME>(S, C, y, yn, [](int, V2, V2) {})) {
#pragma unroll
      for (int q = 0; q < 4; ++q) yn[q] = y[q];
      ok = fp64_rk4(A, yn);
      if (!ok) break;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = yn[q];
  }
  const double nan = NAN;
#pragma unroll
  for (int q = 0; q < 4; ++q) A.end_state[q * A.n + i] = ok ? y[q] : nan;
  A.status[i] = ok ? 0 : 1;
}

// ---------------------------------------------------------------- adjoint --

// The adjoint state is held in units of 2^e, e the exponent of its
// largest component at the start (floats reach from 2^-126 to 2^128, gradients
// can be anything); e = 0 when that is beyond 2^+-900.
__device__ __forceinline__ uint32_t high_word(double v) {
  return static_cast<uint32_t>(bits_of(v) >> 32) & 0x7fffffffu;
}
__device__ __forceinline__ uint32_t largest_word(const double l[4]) {
  return max(max(high_word(l[0]), high_word(l[1])), max(high_word(l[2]), high_word(l[3])));
}
__device__ __forceinline__ uint32_t unit_of(const double l[4]) {
  const uint32_t e = largest_word(l) >> 20;
  return (e > 123 && e < 1923 ? e : 1023u) << 20;
}
// Whether a step may use the pairs: the largest between 2^-60 and 2^60 units,
// or all of them zero.
__device__ __forceinline__ bool in_units(const double l[4]) {
  const uint32_t w = largest_word(l);
  const uint64_t any = bits_of(l[0]) | bits_of(l[1]) | bits_of(l[2]) | bits_of(l[3]);
  return (w > (963u << 20) && w < (1083u << 20)) || (any << 1) == 0;
}

// Sums of pairs over the stages a ray spends in a cell, exact but for the
// third words' rounding (as pairs they lost 2^-48 of the sum at every addition:
// 4.6 times the FP64 kernels' error in the node gradients of u, for 7% less
// time).
struct Sum2 {
  V h, l, m;
};
__device__ __forceinline__ void add_to(Sum2 &a, V2 b) {
  const V2 s = two_sum(a.h, b.h), t = two_sum(a.l, b.l), r = two_sum(t.h, s.l);
  a.h = s.h;
  a.l = r.h;
  a.m = vadd(a.m, vadd(t.l, r.l));
}
__device__ __forceinline__ double sum_of(float h, float l, float m) {
  const F2 s = fast_two_sum(h, l);
  return f2d_zero(s.h) + f2d_zero(s.l + m);
}

// Gradients of one bathymetry and one current cell in the basis of the
// bilinear coefficients (c0, cx, cy, cxy); added to the four nodes (v00 = c0 -
// cx - cy + cxy, v10 = cx - cxy, v01 = cy - cxy, v11 = cxy) when the ray moves
// on.
struct PairAcc {
  int bkey, ckey;   // cells (j (nx - 1) + i), -1: empty
  Sum2 d0, d1;           // depth: (c0, cx), (cy, cxy)
  Sum2 w0, wx, wy, wxy;  // (u, v)
  uint32_t unit_hi; // high word of the power of two the sums are in units of
  __device__ __forceinline__ double unit() const { return double_of(unit_hi, 0u); }
  __device__ __forceinline__ double per_unit() const { return double_of(0x7fe00000u - unit_hi, 0u); }
};

__device__ __forceinline__ Sum2 empty_sum() {
  const V z = both(0.0f);
  return Sum2{z, z, z};
}
__device__ __forceinline__ void clear_bathy(PairAcc &a) { a.d0 = a.d1 = empty_sum(); }
__device__ __forceinline__ void clear_current(PairAcc &a) {
  a.w0 = a.wx = a.wy = a.wxy = empty_sum();
}
__device__ __forceinline__ double x_sum(const Sum2 &a) { return sum_of(a.h.x, a.l.x, a.m.x); }
__device__ __forceinline__ double y_sum(const Sum2 &a) { return sum_of(a.h.y, a.l.y, a.m.y); }

__device__ __forceinline__ void nodes_of(double c0, double cx, double cy, double cxy,
                                         double v[4]) {
  v[3] = cxy;
  v[1] = cx - cxy;
  v[2] = cy - cxy;
  v[0] = (c0 - cx) + (cxy - cy);
}

__device__ __forceinline__ int64_t node_of(int key, int nx) {
  return static_cast<int64_t>(key / (nx - 1)) * nx + key % (nx - 1);
}

__device__ __noinline__ void scatter_nodes(double *arr, int64_t base, int nx, uint32_t unit_hi,
                                           double v0, double v1, double v2, double v3) {
  const double u = double_of(unit_hi, 0u);
  const double v[4] = {v0 * u, v1 * u, v2 * u, v3 * u};
  scatter4<double>(arr, base, nx, v);
}

__device__ __forceinline__ void add_nodes(double *arr, int64_t base, int nx, uint32_t unit_hi,
                                          const double v[4]) {
  scatter_nodes(arr, base, nx, unit_hi, v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void flush_bathy(const SplitArgs &S, PairAcc &a) {
  if (a.bkey >= 0) {
    double v[4];
    nodes_of(x_sum(a.d0), y_sum(a.d0), x_sum(a.d1), y_sum(a.d1), v);
    add_nodes(S.A.grad_depth, node_of(a.bkey, S.b.nx), S.b.nx, a.unit_hi, v);
  }
  a.bkey = -1;
  clear_bathy(a);
}

__device__ __forceinline__ void flush_current(const SplitArgs &S, PairAcc &a) {
  if (a.ckey >= 0) {
    const int64_t base = node_of(a.ckey, S.c.nx);
    double v[4];
    nodes_of(x_sum(a.w0), x_sum(a.wx), x_sum(a.wy), x_sum(a.wxy), v);
    add_nodes(S.A.grad_u, base, S.c.nx, a.unit_hi, v);
    nodes_of(y_sum(a.w0), y_sum(a.wx), y_sum(a.wy), y_sum(a.wxy), v);
    add_nodes(S.A.grad_v, base, S.c.nx, a.unit_hi, v);
  }
  a.ckey = -1;
  clear_current(a);
}

// The anchor of M: in FP64 at a state, and the same in pairs.
struct MAnchor {
  double w, beta, kx, ky;
  F2 wp, bp;
  V2 kv;
};

__device__ __forceinline__ F2 beta_of(const Wave &wv, const Eqs &e) {
  return mul(add(e.qk, neg(e.w)), sqr(wv.rk));
}
// w x + beta (k . x) k
__device__ __forceinline__ V2 apply_m(F2 w, F2 beta, V2 kv, V2 x) {
  return add(mul(both(w), x), mul(both(mul(beta, sum_lanes(mul(kv, x)))), kv));
}

// One stage's transpose: rx, and rk less the anchor's M wx; the node
// gradients of (wx, wk) . F added to acc.
template <bool SAME>
__device__ __forceinline__ void stage_vjp(const SplitArgs &S, const DiffCell &C, const Wave &wv,
                                          const At &p, const Eqs &e, const MAnchor &M, V2 wx,
                                          V2 wk, V2 *rx, V2 *rk, PairAcc &acc) {
  if (C.bkey != acc.bkey) {
    flush_bathy(S, acc);
    acc.bkey = C.bkey;
  }
  if (C.ckey != acc.ckey) {
    flush_current(S, acc);
    acc.ckey = C.ckey;
  }
  const V2 kb = mul(wk, S.b.inv);                 // wk over the spacing, per grid
  const V2 kc = SAME ? kb : mul(wk, S.c.inv);
  const V2 g = V2{V{C.b[0].y, C.b[0].z}, V{C.b[1].y, C.b[1].z}};
  const F2 gamma = sum_lanes(mul(kb, g));         // wk . grad h
  const F2 alpha = sum_lanes(mul(wx, wv.kv));     // wx . k
  const F2 qhr = mul(e.qh, wv.rk);                // c_g,h / k
  const F2 gh = add(mul(alpha, qhr), mul(gamma, e.fh));
  // position
  const V2 hxy = mul(lanes(p.hx, p.hy), S.b.inv);
  const F2 ux = sum_lanes(mul(wx, p.wx)), uy = sum_lanes(mul(wx, p.wy));
  *rx = add(mul(both(gh), hxy), mul(lanes(ux, uy), S.c.inv));
  // wavenumber: M wx - c_g,h / k gamma k - (wk . grad u, wk . grad v)
  const F2 beta = beta_of(wv, e);
  const F2 kk = add(mul(beta, alpha), neg(mul(qhr, gamma)));
  V2 r = add(mul(both(e.w), wx), mul(both(kk), wv.kv));
  r = sub(r, apply_m(M.wp, M.bp, M.kv, wx));
  const V2 kcx = both(x_of(kc)), kcy = both(y_of(kc));
  *rk = sub(r, add(mul(kcx, C.wx()), mul(kcy, C.wy())));
  // nodes
  const F2 fx = x_of(p.fb), fy = y_of(p.fb);
  const V2 fk = mul(both(e.f), kb);
  const F2 ghx = mul(gh, fx);
  add_to(acc.d0, lanes(gh, add(ghx, x_of(fk))));
  add_to(acc.d1, lanes(add(mul(gh, fy), y_of(fk)), mul(ghx, fy)));
  const V2 gx = both(x_of(p.fc)), gy = both(y_of(p.fc));
  const V2 wfx = mul(wx, gx);
  add_to(acc.w0, wx);
  add_to(acc.wx, sub(wfx, mul(wv.kv, kcx)));
  add_to(acc.wy, sub(mul(wx, gy), mul(wv.kv, kcy)));
  add_to(acc.wxy, mul(wfx, gy));
}

// M's anchor at a state; false where the pairs do not cover it.
template <bool SAME>
__device__ __noinline__ bool anchor_at(const SplitArgs &S, const double *yin, MAnchor *M) {
  const double y[4] = {yin[0], yin[1], yin[2], yin[3]};
  Base b, c;
  DiffCell C;
  if (!base_of(S.b, y[0], y[1], &b)) return false;
  if (!SAME && !base_of(S.c, y[0], y[1], &c)) return false;
  At p;
  take_cells<SAME>(S, b.i, b.j, SAME ? 0 : c.i, SAME ? 0 : c.j, C);
  fields_at<SAME>(C, b.f, SAME ? b.f : c.f, &p);
  const Wave wv = wave_of(lanes(to_pair(y[2]), to_pair(y[3])));
  if (!diff_ok(p, wv.k2.h)) return false;
  Eqs e;
  double w64, beta64;
  eqs_of<true>(wv, p.h, &e, true, y[2], y[3], depth64(S, b), &w64, &beta64);
  *M = MAnchor{w64, beta64, y[2], y[3], e.w, beta_of(wv, e), wv.kv};
  return true;
}

// A step backward in FP64 (diff.cu), its stage states recomputed from y; the
// node gradients go straight to the arrays.  False (nothing added) where a
// stage has no derivative.
__device__ __noinline__ bool fp64_reverse(const DiffArgs<double> &A, const double *y0,
                                          double *lam_io) {
  Point<double> P;
  double Y[4][4], kd[4], w[4], r[4], lam[4], sum[4];
  const double h = A.dt, half = h * 0.5;
#pragma unroll
  for (int q = 0; q < 4; ++q) { Y[0][q] = y0[q]; lam[q] = lam_io[q]; sum[q] = 0.0; }
  for (int st = 0; st < 3; ++st) {
    if (!eval(A, Y[st], P, kd)) return false;
    for (int q = 0; q < 4; ++q) Y[st + 1][q] = y0[q] + kd[q] * (st == 2 ? h : half);
  }
  if (!eval(A, Y[3], P, kd)) return false;
  NodeAcc<double> acc;
  acc.bkey = acc.ckey = -1;
#pragma unroll
  for (int q = 0; q < 4; ++q) acc.d[q] = acc.u[q] = acc.v[q] = r[q] = 0.0;
  for (int st = 3; st >= 0; --st) {
    if (st < 3) eval(A, Y[st], P, kd);
    const double c = (st == 0 || st == 3) ? h / 6.0 : h / 3.0;
    const double f = st == 3 ? 0.0 : st == 2 ? h : half;
    for (int q = 0; q < 4; ++q) w[q] = lam[q] * c + f * r[q];
    vjp(A, Y[st], P, w, r, acc);
    for (int q = 0; q < 4; ++q) sum[q] += r[q];
  }
  flush_bathy(A, acc);
  flush_current(A, acc);
  for (int q = 0; q < 4; ++q) lam_io[q] = lam[q] + sum[q];
  return true;
}

template <bool SAME>
__global__ void __launch_bounds__(kSplitBlock, 4)
    diff_split_adjoint(const __grid_constant__ SplitArgs S) {
  const DiffArgs<double> &A = S.A;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  if (A.status[i] != 0) {  // no gradient through a ray that stopped
#pragma unroll
    for (int q = 0; q < 4; ++q) A.grad_state0[q * A.n + i] = 0.0;
    return;
  }
  double lam[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) lam[q] = A.grad_end[q * A.n + i];
  PairAcc acc;
  acc.bkey = acc.ckey = -1;
  clear_bathy(acc);
  clear_current(acc);
  acc.unit_hi = unit_of(lam);
#pragma unroll
  for (int q = 0; q < 4; ++q) lam[q] *= acc.per_unit();
  DiffCell C;
  MAnchor M{};
  bool anchored = false;
  // Scratch of a step, 16 doubles a ray: the state y (4), then per stage 2-4
  // displacement and wavenumber (x and y) as pairs, a pair in a double's
  // place.  A step of the FP64 form is marked by a NaN displacement.
  float2 *const pairs = reinterpret_cast<float2 *>(A.seg);
  for (int64_t seg = A.n_ck - 1; seg >= 0; --seg) {
    const int64_t first = seg * A.ck_every;
    const int64_t last = min(first + A.ck_every, A.steps);  // steps [first, last)
    double y[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = A.ckpt[(seg * 4 + q) * A.n + i];
    for (int64_t s = first; s < last; ++s) {
      const int64_t row = (s - first) * 16 * A.n + i;
#pragma unroll
      for (int q = 0; q < 4; ++q) A.seg[row + q * A.n] = y[q];
      double yn[4];
      const bool ok = forward_step<SAME>(S, C, y, yn, [&](int st, V2 disp, V2 q) {
        float2 *p = pairs + row + (4 + 4 * st) * A.n;
        p[0] = make_float2(disp.h.x, disp.l.x);
        p[A.n] = make_float2(disp.h.y, disp.l.y);
        p[2 * A.n] = make_float2(q.h.x, q.l.x);
        p[3 * A.n] = make_float2(q.h.y, q.l.y);
      });
      if (!ok) {
        pairs[row + 4 * A.n] = make_float2(NAN, NAN);
#pragma unroll
        for (int q = 0; q < 4; ++q) yn[q] = y[q];
        if (!fp64_rk4(A, yn)) goto done;  // (diff.cu)
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) y[q] = yn[q];
    }
    // The segment backward.  M's anchor for a step is its new state: the
    // first stage of the step handled before, or of the rays' end.
    if (seg == A.n_ck - 1) {
      double yv[4] = {y[0], y[1], y[2], y[3]};
      MAnchor m;
      anchored = anchor_at<SAME>(S, yv, &m);
      M = m;
    }
    for (int64_t s = last - 1; s >= first; --s) {
      const int64_t row = (s - first) * 16 * A.n + i;
#pragma unroll
      for (int q = 0; q < 4; ++q) y[q] = A.seg[row + q * A.n];
      Base b, c;
      bool split = !isnan(pairs[row + 4 * A.n].x) && in_units(lam) && base_of(S.b, y[0], y[1], &b) &&
                   (SAME || base_of(S.c, y[0], y[1], &c));
      if (split && !anchored) {  // after a step of the FP64 form
        double yv[4] = {y[0], y[1], y[2], y[3]};
        MAnchor m;
        split = anchor_at<SAME>(S, yv, &m);
        M = m;
      }
      if (!split) {
        double yv[4] = {y[0], y[1], y[2], y[3]}, lv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) lv[q] = lam[q] * acc.unit();
        if (!fp64_reverse(A, yv, lv)) goto done;
#pragma unroll
        for (int q = 0; q < 4; ++q) lam[q] = lv[q] * acc.per_unit();
        anchored = false;
        continue;
      }
      // the stages' weights of lam are dt/6 and twice that
      const V2 lx = lanes(to_pair(lam[0] * S.sixth), to_pair(lam[1] * S.sixth));
      const V2 lk = lanes(to_pair(lam[2] * S.sixth), to_pair(lam[3] * S.sixth));
      V2 rx = zero2(), rk = rx;         // the later stage's r (rk: all of it)
      V2 sx = rx, sk = rx, ox = rx;     // sums of rx, of rk less M wx, of wx less lx's part
      const double h64 = depth64(S, b);
      MAnchor next;  // set by the first stage, handled last
#pragma unroll 1
      for (int st = 3; st >= 0; --st) {
        // wx, wk = c lam + f r of the stage after
        const float cw = st == 3 || st == 0 ? 1.0f : 2.0f;
        V2 wx = scale(cw, lx), wk = scale(cw, lk);
        if (st < 3) {
          const V2 f = both(st == 2 ? S.dt2 : S.half2);
          const V2 dx = mul(rx, f);
          ox = add(ox, dx);
          wx = add(wx, dx);
          wk = add(wk, mul(rk, f));
        }
        Wave wv;
        At p;
        V2 disp = zero2(), q;
        if (st == 0) {
          y[2] = A.seg[row + 2 * A.n];  // again: not held through the stages
          y[3] = A.seg[row + 3 * A.n];
          q = lanes(to_pair(y[2]), to_pair(y[3]));
        } else {
          const float2 *t = pairs + row + 4 * st * A.n;
          const float2 t0 = t[0], t1 = t[A.n], t2 = t[2 * A.n], t3 = t[3 * A.n];
          disp = V2{V{t0.x, t1.x}, V{t0.y, t1.y}};
          q = V2{V{t2.x, t3.x}, V{t2.y, t3.y}};
        }
        wv = wave_of(q);
        (void)stage_at<SAME>(S, b, c, disp, C, &p);
        Eqs e;
        const bool anchor = st == 0;
        eqs_of<true>(wv, p.h, &e, anchor, y[2], y[3], h64, &next.w, &next.beta);
        if (anchor) {
          next.wp = e.w;
          next.bp = beta_of(wv, e);
          next.kv = wv.kv;
        }
        V2 dk;
        stage_vjp<SAME>(S, C, wv, p, e, M, wx, wk, &rx, &dk, acc);
        rk = add(dk, apply_m(M.wp, M.bp, M.kv, wx));
        sx = add(sx, rx);
        sk = add(sk, dk);
      }
      // lam_k += M (sum of wx) in FP64 + the pairs' differences; the sum of
      // the stages' wx is dt lam_x + ox
      const double gx = fma(A.dt, lam[0], to_double(x_of(ox)));
      const double gy = fma(A.dt, lam[1], to_double(y_of(ox)));
      const double kg = M.beta * fma(M.kx, gx, M.ky * gy);
      lam[0] += to_double(x_of(sx));
      lam[1] += to_double(y_of(sx));
      lam[2] += fma(M.w, gx, kg * M.kx) + to_double(x_of(sk));
      lam[3] += fma(M.w, gy, kg * M.ky) + to_double(y_of(sk));
      M = next;
      M.kx = y[2];
      M.ky = y[3];
      anchored = true;
    }
  }
done:
  flush_bathy(S, acc);
  flush_current(S, acc);
#pragma unroll
  for (int q = 0; q < 4; ++q) A.grad_state0[q * A.n + i] = lam[q] * acc.unit();
}

// ---------------------------------------------------------------- tangent --

// The tangent form's own arguments: the tangent fields' records, as those of
// the fields but each cell's (u's and v's apart) in units of 2^e, e the
// exponent of its largest coefficient, and that exponent as in a double's high
// word (0: all zero; kNoRecord: not finite, or beyond 2^+-850).  Null: none.
//
// Tangents have no natural size, and those of one call may span any range (a
// fill value at a node no ray meets, one ray among many), so each step of each
// ray has a unit too, a power of two near the largest component of its tangent
// (while that is 0: its cells' largest coefficient), and the pairs hold values
// in that unit.  A step is on pairs where, in units,
//   each component of the ray's tangent is 0 or at least 2^-100 (below, its
//   pair loses the low half), and
//   each cell's largest coefficient is 0, or 2^-72 to 2^120 (what the smaller
//   ones lose, 2^-124, is then below the rounding of the nodes' differences),
//   or less where every component of the ray's tangent is 2^-30 or more (and
//   that loss is below its rounding);
// every other step, and one whose result is not finite, runs in FP64.
struct TangentArgs {
  SplitArgs S;
  const float4 *db, *dc;
  const uint32_t *db_e;
  const uint2 *dc_e;
};
constexpr uint32_t kNoRecord = 0x7ff00000u;

// The cells of the tangent fields that a lane holds, in units; tiny: a
// coefficient field is nonzero and below 2^-72 units, bad: not covered.
struct TangentCell : DiffCell {
  bool b_tiny = false, b_bad = false, c_tiny = false, c_bad = false;
};

// Order of magnitude: the high word, at least 1 for anything but 0.
__device__ __forceinline__ uint32_t magnitude_word(double v) {
  return high_word(v) | (static_cast<uint32_t>(bits_of(v)) != 0u ? 1u : 0u);
}
__device__ __forceinline__ uint32_t exponent_word(const double o[4]) {
  const uint32_t w = max(max(magnitude_word(o[0]), magnitude_word(o[1])),
                         max(magnitude_word(o[2]), magnitude_word(o[3])));
  return w == 0 || (w >= (173u << 20) && w < (1873u << 20)) ? w & 0x7ff00000u : kNoRecord;
}

// A unit is given as `sh`: its exponent, in place to be added to a high word.
// v is below 2^127 units.  split3's parts, with a low half down to 2^-149.
__device__ __forceinline__ F2 pair_in_units(double v, int32_t sh) {
  const uint32_t hi = static_cast<uint32_t>(bits_of(v) >> 32), lo = static_cast<uint32_t>(bits_of(v));
  const uint32_t sign = hi & 0x80000000u;
  const int32_t e = static_cast<int32_t>((hi >> 20) & 0x7ffu) - (sh >> 20) - 1023;
  const float h = float_of(sign | static_cast<uint32_t>(e + 127) << 23 | (hi & 0xfffffu) << 3 | lo >> 29);
  // the 29 bits after, in units of 2^(e - 52)
  const uint32_t n = lo & 0x1fffffffu;
  const float t = fma32(float_of(0x4b000000u | n >> 6) - 8388608.0f, 64.0f,
                        float_of(0x4b000000u | (n & 63u)) - 8388608.0f);
  const float l = (t * 0x1p-26f) * float_of(sign | static_cast<uint32_t>(e - 26 + 127) << 23);
  return F2{e < -126 ? 0.0f : h, e < -100 ? 0.0f : l};
}
__device__ __forceinline__ double from_units(float f, int32_t sh) {
  if (f == 0.0f) return 0.0;
  const uint64_t b = bits_of(f2d_normal(f));
  return double_of(static_cast<uint32_t>(b >> 32) + static_cast<uint32_t>(sh),
                   static_cast<uint32_t>(b));
}
// On the floats: their conversions to doubles make infinities and NaN finite.
__device__ __forceinline__ bool all_finite(V2 a) {
  const V s = vadd(a.h, a.l);
  return fabsf(s.x) < 0x1p126f && fabsf(s.y) < 0x1p126f;
}

__global__ void build_tangent_records(TangentArgs T, float4 *db, float4 *dc, uint32_t *db_e,
                                      uint2 *dc_e) {
  const DiffArgs<double> &A = T.S.A;
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  auto unit = [](uint32_t w) {
    return w == 0 || w == kNoRecord ? 0 : static_cast<int32_t>(w) - (1023 << 20);
  };
  if (db && k < static_cast<int64_t>(A.bg.nx - 1) * (A.bg.ny - 1)) {
    double o[4];
    F2 q[4];
    coefficients(A.d_depth, A.bg.nx, k, o);
    const uint32_t w = exponent_word(o);
    db_e[k] = w;
    for (int t = 0; t < 4; ++t)
      q[t] = w == kNoRecord ? F2{0.0f, 0.0f} : pair_in_units(o[t], unit(w));
    db[2 * k] = make_float4(q[0].h, q[1].h, q[2].h, q[3].h);
    db[2 * k + 1] = make_float4(q[0].l, q[1].l, q[2].l, q[3].l);
  }
  if (dc && k < static_cast<int64_t>(A.cg.nx - 1) * (A.cg.ny - 1)) {
    double o[4] = {0.0, 0.0, 0.0, 0.0}, p[4] = {0.0, 0.0, 0.0, 0.0};
    F2 q[4], r[4];
    if (A.d_u) coefficients(A.d_u, A.cg.nx, k, o);
    if (A.d_v) coefficients(A.d_v, A.cg.nx, k, p);
    const uint32_t wu = exponent_word(o), wv = exponent_word(p);
    dc_e[k] = make_uint2(wu, wv);
    for (int t = 0; t < 4; ++t) {
      q[t] = wu == kNoRecord ? F2{0.0f, 0.0f} : pair_in_units(o[t], unit(wu));
      r[t] = wv == kNoRecord ? F2{0.0f, 0.0f} : pair_in_units(p[t], unit(wv));
    }
    dc[4 * k] = make_float4(q[0].h, r[0].h, q[1].h, r[1].h);
    dc[4 * k + 1] = make_float4(q[2].h, r[2].h, q[3].h, r[3].h);
    dc[4 * k + 2] = make_float4(q[0].l, r[0].l, q[1].l, r[1].l);
    dc[4 * k + 3] = make_float4(q[2].l, r[2].l, q[3].l, r[3].l);
  }
}

// One stage's tangent of (dx, dk): m = M dk, t = m + the rest, and tk.
template <bool SAME>
__device__ __forceinline__ void stage_jvp(const SplitArgs &S, const DiffCell &C, const DiffCell &D,
                                          bool depth, bool current, const Wave &wv, const At &p,
                                          const Eqs &e, V2 dx, V2 dk, V2 *m, V2 *t, V2 *tk) {
  F2 dh = sum_lanes(mul(mul(lanes(p.hx, p.hy), S.b.inv), dx));
  const V2 dc = mul(dx, S.c.inv);
  V2 duv = add(mul(p.wx, both(x_of(dc))), mul(p.wy, both(y_of(dc))));
  At q;
  if (depth || current) fields_at<SAME>(D, p.fb, p.fc, &q);
  if (depth) dh = add(dh, q.h);
  if (current) duv = add(duv, q.uv);
  const F2 alpha = sum_lanes(mul(wv.kv, dk));
  const F2 qhr = mul(e.qh, wv.rk);
  *m = add(mul(both(e.w), dk), mul(both(mul(beta_of(wv, e), alpha)), wv.kv));
  *t = add(*m, add(mul(both(mul(qhr, dh)), wv.kv), duv));
  const F2 df = add(mul(e.fh, dh), neg(mul(qhr, alpha)));
  V2 g = mul(both(df), V2{V{C.b[0].y, C.b[0].z}, V{C.b[1].y, C.b[1].z}});
  if (depth) g = add(g, mul(both(e.f), V2{V{D.b[0].y, D.b[0].z}, V{D.b[1].y, D.b[1].z}}));
  F2 tx = sum_lanes(mul(dk, C.wx())), ty = sum_lanes(mul(dk, C.wy()));
  if (current) {
    tx = add(tx, sum_lanes(mul(wv.kv, D.wx())));
    ty = add(ty, sum_lanes(mul(wv.kv, D.wy())));
  }
  *tk = sub(mul(g, S.b.inv), mul(lanes(tx, ty), S.c.inv));
}

// A record's factor into units of sh, its exponent w (0 where that is below a
// float's, which is used only where tiny is allowed).
__device__ __forceinline__ float unit_factor(uint32_t w, int32_t sh, bool *tiny, bool *bad) {
  const int32_t d = static_cast<int32_t>(w >> 20) - (sh >> 20) - 1023;
  *bad |= d > 120;
  *tiny |= w != 0 && d < -72;
  return w == 0 || d < -126 || d > 120 ? 0.0f : float_of(static_cast<uint32_t>(d + 127) << 23);
}
__device__ __forceinline__ float4 scaled(float4 a, float f, float g) {  // lanes x, z and y, w
  return make_float4(a.x * f, a.y * g, a.z * f, a.w * g);
}

// The tangent fields' cells of a stage, those the lane holds in C; false where
// the pairs do not cover them.  full: every component of the ray's tangent is
// 2^-30 units or more.
__device__ __forceinline__ bool take_tangent_cells(const TangentArgs &T, const DiffCell &C,
                                                   int32_t sh, bool full, TangentCell &D) {
  if (T.db && D.bkey != C.bkey) {
    const float4 *p = T.db + static_cast<int64_t>(C.bkey) * 2;
    D.b_tiny = D.b_bad = false;
    const float f = unit_factor(__ldg(T.db_e + C.bkey), sh, &D.b_tiny, &D.b_bad);
    D.b[0] = scaled(ld4(p), f, f);
    D.b[1] = scaled(ld4(p + 1), f, f);
    D.bkey = C.bkey;
  }
  if (T.dc && D.ckey != C.ckey) {
    const float4 *p = T.dc + static_cast<int64_t>(C.ckey) * 4;
    const uint2 w = __ldg(T.dc_e + C.ckey);
    D.c_tiny = D.c_bad = false;
    const float f = unit_factor(w.x, sh, &D.c_tiny, &D.c_bad);
    const float g = unit_factor(w.y, sh, &D.c_tiny, &D.c_bad);
#pragma unroll
    for (int q = 0; q < 4; ++q) D.c[q] = scaled(ld4(p + q), f, g);
    D.ckey = C.ckey;
  }
  return !(D.b_bad || D.c_bad) && (full || !(D.b_tiny || D.c_tiny));
}

// The unit of a step of tangent dy from the point b, c: the last step's while
// it is within 2^30 of dy's largest component.  False where the pairs do not
// cover dy.
template <bool SAME>
__device__ __forceinline__ bool choose_unit(const TangentArgs &T, const Base &b, const Base &c,
                                            const double dy[4], int32_t *sh, bool *full,
                                            TangentCell &D) {
  uint32_t w[4], top = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    w[q] = magnitude_word(dy[q]);
    top = max(top, w[q]);
  }
  if (top == 0) {
    if (T.db) top = __ldg(T.db_e + (b.j * (T.S.b.nx - 1) + b.i));
    if (T.dc) {
      const Base &g = SAME ? b : c;
      const uint2 e = __ldg(T.dc_e + (g.j * (T.S.c.nx - 1) + g.i));
      top = max(top, max(e.x, e.y));
    }
    if (top == 0) top = 1023u << 20;  // nothing but zeros
  }
  if (top < (173u << 20) || top >= (1873u << 20)) return false;
  const bool change = static_cast<int32_t>(top) < (993 << 20) + *sh ||
                      static_cast<int32_t>(top) > (1053 << 20) + *sh;
  *sh = change ? static_cast<int32_t>(top & 0x7ff00000u) - (1023 << 20) : *sh;
  D.bkey = change ? -1 : D.bkey;
  D.ckey = change ? -1 : D.ckey;
  bool ok = true;
  *full = true;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int32_t m = static_cast<int32_t>(w[q]) - *sh;
    ok &= w[q] == 0 || m >= (923 << 20);
    *full &= w[q] != 0 && m >= (993 << 20);
  }
  return ok;
}

// A step of the state and its tangent; false (y and dy as they were) when a
// stage is outside the pairs' domain.  sh: the unit, kept from step to step.
template <bool SAME>
__device__ __forceinline__ bool tangent_step(const TangentArgs &T, DiffCell &C, TangentCell &D,
                                             int32_t &sh, double y[4], double dy[4]) {
  const SplitArgs &S = T.S;
  Base b, c;
  if (!base_of(S.b, y[0], y[1], &b)) return false;
  if (!SAME && !base_of(S.c, y[0], y[1], &c)) return false;
  const V2 k = lanes(to_pair(y[2]), to_pair(y[3]));
  const bool depth = T.db != nullptr, current = T.dc != nullptr;
  bool full;
  if (!choose_unit<SAME>(T, b, c, dy, &sh, &full, D)) return false;
  const V2 dx0 = lanes(pair_in_units(dy[0], sh), pair_in_units(dy[1], sh));
  const V2 dk0 = lanes(pair_in_units(dy[2], sh), pair_in_units(dy[3], sh));
  V2 disp = zero2(), q = k, dx = dx0, dq = dk0;       // the stage's state
  V2 d1 = disp, k1 = disp, m1 = disp, sd = disp, sk = disp, sdx = disp, sdk = disp;
  double a[4] = {0.0, 0.0, 0.0, 0.0}, mx = 0.0, my = 0.0;  // anchors
#pragma unroll 1
  for (int st = 0; st < 4; ++st) {
    At p;
    if (!stage_at<SAME>(S, b, c, disp, C, &p)) return false;
    if (!take_tangent_cells(T, C, sh, full, D)) return false;
    const Wave wv = wave_of(q);
    if (!diff_ok(p, wv.k2.h)) return false;
    Eqs e;
    Fields64 F{};
    double w64 = 0.0, beta64 = 0.0, f64 = 0.0;
    if (st == 0) F = fields64<SAME>(S, b, c);
    eqs_of<true>(wv, p.h, &e, st == 0, y[2], y[3], F.h, &w64, &beta64, &f64);
    V2 d, dk, m, t, tk;
    derivative(S, C, wv, p, e, &d, &dk);
    stage_jvp<SAME>(S, C, D, depth, current, wv, p, e, dx, dq, &m, &t, &tk);
    if (st == 0) {
      anchors(F, y, w64, f64, a);
      const double kg = beta64 * fma(y[2], dy[2], y[3] * dy[3]);
      mx = fma(w64, dy[2], kg * y[2]);
      my = fma(w64, dy[3], kg * y[3]);
      d1 = d;
      m1 = m;
      k1 = dk;
      sdx = sub(t, m);
      sdk = tk;
    } else {
      const float wt = st == 3 ? 1.0f : 2.0f;
      sd = add(sd, scale(wt, sub(d, d1)));
      sk = add(sk, scale(wt, sub(dk, k1)));
      sdx = add(sdx, scale(wt, sub(t, m1)));
      sdk = add(sdk, scale(wt, tk));
    }
    const V2 hs = both(st == 2 ? S.dt2 : S.half2);
    disp = mul(d, hs);
    q = add(k, mul(dk, hs));
    dx = add(dx0, mul(t, hs));
    dq = add(dk0, mul(tk, hs));
  }
  const V2 s6 = mul(sd, both(S.sixth2)), k6 = mul(sk, both(S.sixth2));
  const V2 t6 = mul(sdx, both(S.sixth2));
  if (!(all_finite(t6) && all_finite(sdk))) return false;
  y[0] += fma(S.A.dt, a[0], f2d_zero(s6.h.x)) + f2d_zero(s6.l.x);
  y[1] += fma(S.A.dt, a[1], f2d_zero(s6.h.y)) + f2d_zero(s6.l.y);
  y[2] += fma(S.A.dt, a[2], f2d_zero(k6.h.x)) + f2d_zero(k6.l.x);
  y[3] += fma(S.A.dt, a[3], f2d_zero(k6.h.y)) + f2d_zero(k6.l.y);
  dy[0] += fma(S.A.dt, mx, from_units(t6.h.x, sh)) + from_units(t6.l.x, sh);
  dy[1] += fma(S.A.dt, my, from_units(t6.h.y, sh)) + from_units(t6.l.y, sh);
  dy[2] = fma(S.sixth, from_units(sdk.h.x, sh) + from_units(sdk.l.x, sh), dy[2]);
  dy[3] = fma(S.sixth, from_units(sdk.h.y, sh) + from_units(sdk.l.y, sh), dy[3]);
  return true;
}

// A step in FP64 (diff.cu), state and tangent; false when the ray stops.
__device__ __noinline__ bool fp64_tangent(const DiffArgs<double> &A, double *y, double *dy) {
  double t[4], dt[4], sum[4] = {0.0, 0.0, 0.0, 0.0}, dsum[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 4; ++q) { t[q] = y[q]; dt[q] = dy[q]; }
#pragma unroll 1
  for (int st = 0; st < 4; ++st) {
    Point<double> P;
    double k[4], d[4];
    if (!eval(A, t, P, k)) return false;
    jvp(A, t, P, dt, d);
    const double wt = st == 0 || st == 3 ? 1.0 : 2.0, h = st == 2 ? A.dt : A.dt * 0.5;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      sum[q] = sum[q] + k[q] * wt;
      dsum[q] = dsum[q] + d[q] * wt;
      t[q] = y[q] + k[q] * h;
      dt[q] = dy[q] + d[q] * h;
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    y[q] += sum[q] * (A.dt / 6.0);
    dy[q] += dsum[q] * (A.dt / 6.0);
  }
  return true;
}

template <bool SAME>
__global__ void __launch_bounds__(kSplitBlock)
    diff_split_tangent(const __grid_constant__ TangentArgs T) {
  const DiffArgs<double> &A = T.S.A;
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned lanes_of_warp = __ballot_sync(0xffffffffu, i < A.n);
  if (i >= A.n) return;
  double y[4] = {A.x0[i], A.y0[i], A.kx0[i], A.ky0[i]};
  double dy[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) dy[q] = A.dstate0[q * A.n + i];
  bool ok = true;
  DiffCell C;
  TangentCell D;
  int32_t sh = 0;
  for (int64_t s = 0; s < A.steps; ++s) {
    if (ok && !tangent_step<SAME>(T, C, D, sh, y, dy)) {
      double yv[4], dv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { yv[q] = y[q]; dv[q] = dy[q]; }
      ok = fp64_tangent(A, yv, dv);
#pragma unroll
      for (int q = 0; q < 4; ++q) { y[q] = yv[q]; dy[q] = dv[q]; }
    }
    // Together again: lanes that a step has parted (a new unit, a step in FP64)
    // otherwise stay so to the end, at twice the time.
    if ((s & 7) == 7 && !__any_sync(lanes_of_warp, ok)) break;
  }
  const double nan = NAN;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    A.end_state[q * A.n + i] = ok ? y[q] : nan;
    A.d_end[q * A.n + i] = ok ? dy[q] : nan;
  }
  A.status[i] = ok ? 0 : 1;
}

F2 host_pair(double v) {
  const float h = static_cast<float>(v);
  return F2{h, static_cast<float>(v - static_cast<double>(h))};
}

SplitField field_of(int nx, int ny, double x0, double y0, double inv_dx, double inv_dy) {
  SplitField f{};
  f.nx = nx;
  f.ny = ny;
  f.x0 = x0;
  f.y0 = y0;
  f.inv_dx = inv_dx;
  f.inv_dy = inv_dy;
  const F2 a = host_pair(inv_dx), b = host_pair(inv_dy);
  f.inv = V2{V{a.h, b.h}, V{a.l, b.l}};
  return f;
}

bool in_range(double v) { return v > 0x1p-20 && v < 0x1p20; }

// The pool the records come from, one per device for the process (null: none).
// Apart from the device's default pool, which mr_trace has keep what is freed:
// this one keeps kKeptBytes at most and gives the rest back at the next
// synchronisation.  Mapping memory anew takes a call some 140 us and 150 ps a
// cell, as long as seven steps of few rays.  It does not make one stream wait
// for another to reuse memory.
constexpr uint64_t kKeptBytes = 64ull << 20;
cudaMemPool_t record_pool() {
  static std::mutex mu;
  static std::vector<cudaMemPool_t> pools;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (static_cast<size_t>(device) >= pools.size()) pools.resize(device + 1, nullptr);
  if (!pools[device]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    uint64_t keep = kKeptBytes;
    int no = 0;
    if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return nullptr;
    if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
        cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &no) !=
            cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return nullptr;
    }
    pools[device] = pool;
  }
  return pools[device];
}

}  // namespace

bool launch_diff_split(DiffForm form, const DiffCall &k, cudaStream_t stream, cudaError_t *err) {
  const int64_t bn = static_cast<int64_t>(k.bnx - 1) * (k.bny - 1);
  const int64_t cn = static_cast<int64_t>(k.cnx - 1) * (k.cny - 1);
  const int64_t cells = bn > cn ? bn : cn;
  const bool db = form == DIFF_TANGENT && k.d_depth;
  const bool dc = form == DIFF_TANGENT && (k.d_u || k.d_v);
  const size_t records = static_cast<size_t>(bn) * 64 + static_cast<size_t>(cn) * 128;
  const size_t db_bytes = db ? static_cast<size_t>(bn) * 32 : 0;
  const size_t dc_bytes = dc ? static_cast<size_t>(cn) * 64 : 0;
  const size_t dce_bytes = dc ? static_cast<size_t>(cn) * 8 : 0;
  const size_t dbe_bytes = db ? static_cast<size_t>(bn) * 4 : 0;
  const size_t bytes = records + db_bytes + dc_bytes + dce_bytes + dbe_bytes;
  // Where pairs pay, per pass.  A step on pairs saves 20 us of few rays' FP64
  // chain, 1.6 ns a ray of many rays'.  Against that stand the records: their
  // launch and allocation, 45 us of host and device time for a forward or
  // adjoint pass and 19 for a tangent one (one pass), 40 ps a cell to fill them,
  // and, beyond what the pool keeps, mapping memory.  Adjoint (both passes) and
  // tangent, FP64 -> pairs, us: 217 rays on 200^2 nodes, 1 step 422 / 56 -> 469
  // / 58 (not taken), 5 steps 548 / 180 -> 468 / 100, 100 steps 6,977 / 3,117 ->
  // 3,094 / 1,082; on 1,024^2, 10 steps 834 / 338 -> 931 / 468 (not taken), 20
  // steps 1,508 / 650 -> 1,082 / 489; 32,768 rays there, 5 steps 857 / 361 ->
  // 852 / 435 (not taken), 10 steps 1,565 / 696 -> 942 / 420.  Grids of up to
  // 4,096 cells are on pairs at any length: such a call is the host's time, and
  // the FP64 form's exp(-2 kh) = 1 - (1 - exp(-2 kh)) has few digits from kh = 15
  // on.  Up to 2^24 cells, 5.0 GB of records: what a call may take beside its
  // own buffers.
  if (k.n == 0 || k.steps == 0 || cells > (1ll << 24) || k.bnx > (1 << 20) ||
      k.bny > (1 << 20) || k.cnx > (1 << 20) || k.cny > (1 << 20))
    return false;
  const double per_step = 1.6 * static_cast<double>(k.n);
  const double saved = static_cast<double>(k.steps) * (per_step > 20e3 ? per_step : 20e3);
  const double fixed = form == DIFF_TANGENT || cells <= 4096 ? 19e3 : 45e3;
  const double cost = fixed + (bytes <= kKeptBytes ? 0.04 * static_cast<double>(cells)
                                                   : 120e3 + 0.19 * static_cast<double>(cells));
  if (cost > saved) return false;
  if (!in_range(k.dt) || !in_range(k.b_inv_dx) || !in_range(k.b_inv_dy) ||
      !in_range(k.c_inv_dx) || !in_range(k.c_inv_dy))
    return false;
  SplitArgs S{};
  DiffArgs<double> &A = S.A;
  A.bg = DGrid<double>{k.depth, nullptr, k.bnx, k.bny, k.bx0, k.by0, k.b_inv_dx, k.b_inv_dy};
  A.cg = DGrid<double>{k.u, k.v, k.cnx, k.cny, k.cx0, k.cy0, k.c_inv_dx, k.c_inv_dy};
  A.same_grid = k.same_grid;
  A.n = k.n; A.steps = k.steps; A.ck_every = k.ck_every; A.n_ck = k.n_ck;
  A.x0 = k.x0; A.y0 = k.y0; A.kx0 = k.kx0; A.ky0 = k.ky0;
  A.dt = k.dt;
  A.ckpt = k.ckpt; A.end_state = k.end_state; A.status = k.status;
  A.grad_end = k.grad_end; A.seg = k.seg; A.grad_state0 = k.grad_state0;
  A.grad_depth = k.grad_depth; A.grad_u = k.grad_u; A.grad_v = k.grad_v;
  A.dstate0 = k.dstate0; A.d_depth = k.d_depth; A.d_u = k.d_u; A.d_v = k.d_v;
  A.d_end = k.d_end;
  S.b = field_of(k.bnx, k.bny, k.bx0, k.by0, k.b_inv_dx, k.b_inv_dy);
  S.c = field_of(k.cnx, k.cny, k.cx0, k.cy0, k.c_inv_dx, k.c_inv_dy);
  S.sixth = k.dt / 6.0;
  S.dt2 = host_pair(k.dt);
  S.half2 = host_pair(k.dt * 0.5);
  S.sixth2 = host_pair(S.sixth);
  // Stream-ordered scratch for the records, freed behind the kernels; not
  // while the stream is being captured (the allocation would become a node of
  // the caller's graph).
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  char *mem = nullptr;
  cudaMemPool_t pool = nullptr;
  if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone ||
      !(pool = record_pool()) ||
      cudaMallocFromPoolAsync(reinterpret_cast<void **>(&mem), bytes, pool, stream) !=
          cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  float4 *b = reinterpret_cast<float4 *>(mem);
  double2 *b64 = reinterpret_cast<double2 *>(mem + bn * 32);
  float4 *c = reinterpret_cast<float4 *>(mem + bn * 64);
  double2 *c64 = reinterpret_cast<double2 *>(mem + bn * 64 + cn * 64);
  S.b.rec = b; S.b.rec64 = b64;
  S.c.rec = c; S.c.rec64 = c64;
  build_diff_records<<<static_cast<unsigned>((cells + 255) / 256), 256, 0, stream>>>(S, b, b64, c,
                                                                                     c64);
  const unsigned grid = static_cast<unsigned>((k.n + kSplitBlock - 1) / kSplitBlock);
  if (form == DIFF_FORWARD) {
    if (k.same_grid)
      diff_split_forward<true><<<grid, kSplitBlock, 0, stream>>>(S);
    else
      diff_split_forward<false><<<grid, kSplitBlock, 0, stream>>>(S);
  } else if (form == DIFF_ADJOINT) {
    if (k.same_grid)
      diff_split_adjoint<true><<<grid, kSplitBlock, 0, stream>>>(S);
    else
      diff_split_adjoint<false><<<grid, kSplitBlock, 0, stream>>>(S);
  } else {
    char *p = mem + records;
    float4 *dbr = db ? reinterpret_cast<float4 *>(p) : nullptr;
    float4 *dcr = dc ? reinterpret_cast<float4 *>(p += db_bytes) : nullptr;
    uint2 *dce = dc ? reinterpret_cast<uint2 *>(p += dc_bytes) : nullptr;
    uint32_t *dbe = db ? reinterpret_cast<uint32_t *>(mem + bytes - dbe_bytes) : nullptr;
    const TangentArgs T{S, dbr, dcr, dbe, dce};
    if (db || dc)
      build_tangent_records<<<static_cast<unsigned>((cells + 255) / 256), 256, 0, stream>>>(
          T, dbr, dcr, dbe, dce);
    if (k.same_grid)
      diff_split_tangent<true><<<grid, kSplitBlock, 0, stream>>>(T);
    else
      diff_split_tangent<false><<<grid, kSplitBlock, 0, stream>>>(T);
  }
  *err = cudaGetLastError();
  const cudaError_t f = cudaFreeAsync(mem, stream);
  if (*err == cudaSuccess) *err = f;
  return true;
}

}  // namespace mr
