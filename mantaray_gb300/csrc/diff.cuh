// diff.cuh -- the differentiation form's arguments and its equations and
// partial derivatives in the working precision, included by diff.cu (the
// kernels in that precision) and diff_split.cu (the FP64 kernels on float
// pairs, which leave steps outside the pairs' domain to these).  The model
// and the derivations are described at the top of diff.cu.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/mantaray_gpu.h"
#include "handles.h"

namespace mr {
namespace {

template <typename T>
struct DGrid {
  const T *a;     // depth (bathymetry) or u (current)
  const T *b;     // v (current), null for bathymetry
  int nx, ny;
  T x0, y0, inv_dx, inv_dy;
};

template <typename T>
struct DiffArgs {
  DGrid<T> bg, cg;
  int same_grid;        // the current on the bathymetry's grid: one cell location serves both
  int64_t n;
  const T *x0, *y0, *kx0, *ky0;
  T dt;
  int64_t steps, ck_every, n_ck;
  T *ckpt;              // [n_ck][4][n]
  T *end_state;         // [4][n]
  uint8_t *status;      // [n]
  // adjoint
  const T *grad_end;    // [4][n]
  T *seg;               // [ck_every][16][n]: y and the stage states Y2, Y3, Y4
  T *grad_state0;       // [4][n]
  double *grad_depth;   // [bny*bnx]
  double *grad_u, *grad_v;  // [cny*cnx]
  // tangent
  const T *dstate0;     // [4][n]
  const T *d_depth, *d_u, *d_v;
  T *d_end;             // [4][n]
};

// Fast math helpers per precision.
__device__ __forceinline__ double t_expm1(double x) { return expm1(x); }
__device__ __forceinline__ float t_expm1(float x) { return expm1f(x); }
__device__ __forceinline__ double t_rsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float t_rsqrt(float x) { return rsqrtf(x); }
__device__ __forceinline__ double t_floor(double x) { return floor(x); }
__device__ __forceinline__ float t_floor(float x) { return floorf(x); }

template <typename T>
struct Cell {
  int i, j;
  T fx, fy;
};

// Cell holding (x, y): the reference's corner rule (index in [0, n-1], the
// last cell for index n-1).  False outside the grid or for NaN.
template <typename T>
__device__ __forceinline__ bool locate(const DGrid<T> &g, T x, T y, Cell<T> *c) {
  const T ix = (x - g.x0) * g.inv_dx, iy = (y - g.y0) * g.inv_dy;
  if (!(ix >= T(0) && ix <= T(g.nx - 1) && iy >= T(0) && iy <= T(g.ny - 1))) return false;
  T fi = t_floor(ix), fj = t_floor(iy);
  if (fi > T(g.nx - 2)) fi = T(g.nx - 2);
  if (fj > T(g.ny - 2)) fj = T(g.ny - 2);
  c->i = static_cast<int>(fi);
  c->j = static_cast<int>(fj);
  c->fx = ix - fi;
  c->fy = iy - fj;
  return true;
}

// Bilinear value, its spatial derivatives (already divided by the spacing)
// and the cell forward differences of field `a` in cell c.
template <typename T>
struct Interp {
  T val, dxp, dyp;  // value, d/dx, d/dy of the bilinear surface
  T gx, gy;         // cell forward differences (cell-constant gradient)
};

// Bilinear coefficients (value at the south-west node, differences along x and
// y, cross difference) of field `a` in cell c.
template <typename T>
__device__ __forceinline__ void take_cell(const T *a, const DGrid<T> &g, const Cell<T> &c, T e[4]) {
  const int64_t base = static_cast<int64_t>(c.j) * g.nx + c.i;
  const T v00 = __ldg(a + base), v10 = __ldg(a + base + 1);
  const T v01 = __ldg(a + base + g.nx), v11 = __ldg(a + base + g.nx + 1);
  e[0] = v00;
  e[1] = v10 - v00;
  e[2] = v01 - v00;
  e[3] = ((v11 - v10) - v01) + v00;
}

// The coefficients of the cells a lane was last in: a ray stays in a cell for
// several stages, and fetching 12 nodes at each was what the FP32 adjoint waited
// for (with the registers this takes: 10.9 to 8.0 ms for 131,071 rays x 300
// steps).
template <typename T>
struct Held {
  int bi = -1, bj = -1, ci = -1, cj = -1;
  T h[4], u[4], v[4];
};

template <typename T>
__device__ __forceinline__ Interp<T> interp(const T e[4], const DGrid<T> &g, const Cell<T> &c) {
  const T v00 = e[0], ex = e[1], ey = e[2], exy = e[3];
  Interp<T> r;
  r.val = ((v00 + ex * c.fx) + ey * c.fy) + exy * c.fx * c.fy;
  r.dxp = (ex + exy * c.fy) * g.inv_dx;
  r.dyp = (ey + exy * c.fx) * g.inv_dy;
  r.gx = ex * g.inv_dx;
  r.gy = ey * g.inv_dy;
  return r;
}

// Everything the RHS and its derivatives need at one state.
template <typename T>
struct Point {
  Cell<T> cb, cc;
  Interp<T> h, u, v;
  T k, rk, c, s;         // |k|, 1/|k|, kx/k, ky/k
  T q, q_k, q_h;         // group velocity and its partials
  T f, f_k, f_h;         // refraction factor and its partials
};

constexpr double kG = 9.8;

// Evaluates F at s; false when the reference would produce NaN there
// (outside a grid, depth <= 0, k <= 0, non-finite).  HELD: N has the cells of
// the lane's last call.
template <bool HELD = true, typename T>
__device__ __forceinline__ bool eval(const DiffArgs<T> &A, const T s[4], Point<T> &P, T F[4],
                                     Held<T> &N) {
  if (!locate(A.bg, s[0], s[1], &P.cb)) return false;
  if (A.same_grid)
    P.cc = P.cb;
  else if (!locate(A.cg, s[0], s[1], &P.cc))
    return false;
  if (!HELD || P.cb.i != N.bi || P.cb.j != N.bj) {
    take_cell(A.bg.a, A.bg, P.cb, N.h);
    N.bi = P.cb.i;
    N.bj = P.cb.j;
  }
  if (!HELD || P.cc.i != N.ci || P.cc.j != N.cj) {
    take_cell(A.cg.a, A.cg, P.cc, N.u);
    take_cell(A.cg.b, A.cg, P.cc, N.v);
    N.ci = P.cc.i;
    N.cj = P.cc.j;
  }
  P.h = interp(N.h, A.bg, P.cb);
  P.u = interp(N.u, A.cg, P.cc);
  P.v = interp(N.v, A.cg, P.cc);
  const T h = P.h.val;
  const T k2 = s[2] * s[2] + s[3] * s[3];
  if (!(h > T(0)) || !(k2 > T(0))) return false;
  const T g = T(kG);
  // one expm1, one reciprocal and two rsqrt: m4 = 1 - exp(-4a) = m2 (2 - m2),
  // w = 1 / m4, and 1/k, 1/sigma from rsqrt (exact identities)
  const T rk = t_rsqrt(k2);
  const T k = k2 * rk;
  P.k = k;
  P.rk = rk;
  P.c = s[2] * rk;
  P.s = s[3] * rk;
  const T a = k * h;
  const T m2 = -t_expm1(T(-2) * a);  // 1 - exp(-2a)
  const T E = T(1) - m2;             // exp(-2a)
  const T p = T(2) - m2;             // 1 + exp(-2a)
  const T m4 = m2 * p;               // 1 - exp(-4a)
  const T w = T(1) / m4;
  const T rp = m2 * w;               // 1 / p
  const T th = m2 * rp;              // tanh(a)
  const T sech2 = T(4) * E * rp * rp;
  const T isinh2 = T(2) * E * w;     // 1/sinh(2a)
  const T coth2 = (T(2) - m4) * w;   // coth(2a)
  const T gkt = g * k * th;
  const T rsig = t_rsqrt(gkt);
  const T sigma = gkt * rsig;
  const T hrsig = T(0.5) * rsig;     // 1 / (2 sigma)
  const T hrk = T(0.5) * rk;         // 1 / (2 k)
  const T nfac = T(1) + T(2) * a * isinh2;
  const T dsig_dk = g * (th + a * sech2) * hrsig;
  const T dsig_dh = g * k * k * sech2 * hrsig;
  const T dn_da = T(2) * isinh2 - T(4) * a * coth2 * isinh2;
  P.q = sigma * hrk * nfac;
  P.q_k = hrk * ((dsig_dk - sigma * rk) * nfac + sigma * dn_da * h);
  P.q_h = hrk * (dsig_dh * nfac + sigma * dn_da * k);
  P.f = -k * sigma * isinh2;
  P.f_k = -sigma * isinh2 - k * dsig_dk * isinh2 + T(2) * k * sigma * h * coth2 * isinh2;
  P.f_h = -k * dsig_dh * isinh2 + T(2) * k * k * sigma * coth2 * isinh2;
  F[0] = P.q * P.c + P.u.val;
  F[1] = P.q * P.s + P.v.val;
  F[2] = P.f * P.h.gx - s[2] * P.u.gx - s[3] * P.v.gx;
  F[3] = P.f * P.h.gy - s[2] * P.u.gy - s[3] * P.v.gy;
  const bool ok = isfinite(F[0]) && isfinite(F[1]) && isfinite(F[2]) && isfinite(F[3]);
  return ok;
}

template <typename T>
__device__ __forceinline__ bool eval(const DiffArgs<T> &A, const T s[4], Point<T> &P, T F[4]) {
  Held<T> N;
  return eval<false>(A, s, P, F, N);
}

template <typename T>
__device__ __forceinline__ bool rk4(const DiffArgs<T> &A, T y[4], Held<T> &N) {
  Point<T> P;
  T k1[4], k2[4], k3[4], k4[4], t[4];
  const T half = A.dt * T(0.5);
  if (!eval(A, y, P, k1, N)) return false;
#pragma unroll
  for (int q = 0; q < 4; ++q) t[q] = y[q] + k1[q] * half;
  if (!eval(A, t, P, k2, N)) return false;
#pragma unroll
  for (int q = 0; q < 4; ++q) t[q] = y[q] + k2[q] * half;
  if (!eval(A, t, P, k3, N)) return false;
#pragma unroll
  for (int q = 0; q < 4; ++q) t[q] = y[q] + k3[q] * A.dt;
  if (!eval(A, t, P, k4, N)) return false;
  const T sixth = A.dt / T(6);
#pragma unroll
  for (int q = 0; q < 4; ++q) y[q] = y[q] + (((k1[q] + k2[q] * T(2)) + k3[q] * T(2)) + k4[q]) * sixth;
  return true;
}

// ---------------------------------------------------------------- JVP --

template <typename T>
__device__ __forceinline__ T bilin_d(const T *d, const DGrid<T> &g, const Cell<T> &c, T *dgx,
                                     T *dgy) {
  const int64_t base = static_cast<int64_t>(c.j) * g.nx + c.i;
  const T v00 = __ldg(d + base), v10 = __ldg(d + base + 1);
  const T v01 = __ldg(d + base + g.nx), v11 = __ldg(d + base + g.nx + 1);
  *dgx = (v10 - v00) * g.inv_dx;
  *dgy = (v01 - v00) * g.inv_dy;
  return ((v00 + (v10 - v00) * c.fx) + (v01 - v00) * c.fy) + (((v11 - v10) - v01) + v00) * c.fx * c.fy;
}

// dF for the state tangent ds and the field tangents of A (d_depth, d_u, d_v).
template <typename T>
__device__ __forceinline__ void jvp(const DiffArgs<T> &A, const T s[4], const Point<T> &P,
                                    const T ds[4], T dF[4]) {
  T ddx = 0, ddy = 0, dux = 0, duy = 0, dvx = 0, dvy = 0, dD = 0, dU = 0, dV = 0;
  if (A.d_depth) dD = bilin_d(A.d_depth, A.bg, P.cb, &ddx, &ddy);
  if (A.d_u) dU = bilin_d(A.d_u, A.cg, P.cc, &dux, &duy);
  if (A.d_v) dV = bilin_d(A.d_v, A.cg, P.cc, &dvx, &dvy);
  const T dh = P.h.dxp * ds[0] + P.h.dyp * ds[1] + dD;
  const T du = P.u.dxp * ds[0] + P.u.dyp * ds[1] + dU;
  const T dv = P.v.dxp * ds[0] + P.v.dyp * ds[1] + dV;
  const T dk = P.c * ds[2] + P.s * ds[3];
  const T dc = (P.s * P.s * ds[2] - P.c * P.s * ds[3]) * P.rk;
  const T dsn = (-P.c * P.s * ds[2] + P.c * P.c * ds[3]) * P.rk;
  const T dq = P.q_k * dk + P.q_h * dh;
  const T df = P.f_k * dk + P.f_h * dh;
  dF[0] = dq * P.c + P.q * dc + du;
  dF[1] = dq * P.s + P.q * dsn + dv;
  dF[2] = df * P.h.gx + P.f * ddx - ds[2] * P.u.gx - s[2] * dux - ds[3] * P.v.gx - s[3] * dvx;
  dF[3] = df * P.h.gy + P.f * ddy - ds[2] * P.u.gy - s[2] * duy - ds[3] * P.v.gy - s[3] * dvy;
}

// ---------------------------------------------------------------- VJP --

// Per-ray accumulator of node gradients for one bathymetry cell and one
// current cell, in the working precision; flushed to the FP64 node arrays
// when the ray moves on.
template <typename T>
struct NodeAcc {
  int64_t bkey, ckey;   // flat index of the cells' south-west nodes, -1: empty
  T d[4];               // depth nodes (00, 10, 01, 11)
  T u[4], v[4];
};

// Adds `vals[4]` to nodes (base, base+1, base+nx, base+nx+1) of `arr` in
// FP64, summed first across the active lanes of the warp that flush the same
// ones (of the same array: lanes of several call sites may meet here).  Each
// group's lowest lane (its leader) adds its peers' values in ascending lane
// order; the loop runs once per member of the largest group (all active lanes
// take part in every shuffle, each reading the next member of its own group),
// so lanes flushing distinct cells cost no shuffle at all.
template <typename T>
__device__ __forceinline__ void scatter4(double *arr, int64_t base, int nx, const T vals[4]) {
  const unsigned active = __activemask();
  const unsigned peers = __match_any_sync(active, reinterpret_cast<unsigned long long>(arr + base));
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(peers) - 1;
  const unsigned largest = __reduce_max_sync(active, static_cast<unsigned>(__popc(peers)));
  double v[4] = {double(vals[0]), double(vals[1]), double(vals[2]), double(vals[3])};
  unsigned rest = peers & (peers - 1u);  // the group without its leader
  for (unsigned it = 1; it < largest; ++it) {
    const int src = rest ? __ffs(rest) - 1 : lane;
    rest &= rest - 1u;
    T o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) o[q] = __shfl_sync(active, vals[q], src);
    if (lane == leader && src != lane) {
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] += double(o[q]);
    }
  }
  if (lane == leader) {
    atomicAdd(arr + base, v[0]);
    atomicAdd(arr + base + 1, v[1]);
    atomicAdd(arr + base + nx, v[2]);
    atomicAdd(arr + base + nx + 1, v[3]);
  }
}

template <typename T>
__device__ __forceinline__ void flush_bathy(const DiffArgs<T> &A, NodeAcc<T> &acc) {
  if (acc.bkey >= 0) scatter4(A.grad_depth, acc.bkey, A.bg.nx, acc.d);
  acc.bkey = -1;
#pragma unroll
  for (int q = 0; q < 4; ++q) acc.d[q] = T(0);
}

template <typename T>
__device__ __forceinline__ void flush_current(const DiffArgs<T> &A, NodeAcc<T> &acc) {
  if (acc.ckey >= 0) {
    scatter4(A.grad_u, acc.ckey, A.cg.nx, acc.u);
    scatter4(A.grad_v, acc.ckey, A.cg.nx, acc.v);
  }
  acc.ckey = -1;
#pragma unroll
  for (int q = 0; q < 4; ++q) acc.u[q] = acc.v[q] = T(0);
}

// r = J(s)^T w, and the node gradients of w . F added to acc.
template <typename T>
__device__ __forceinline__ void vjp(const DiffArgs<T> &A, const T s[4], const Point<T> &P,
                                    const T w[4], T r[4], NodeAcc<T> &acc) {
  const T c = P.c, sn = P.s;
  const T g_h = (w[0] * c + w[1] * sn) * P.q_h + (w[2] * P.h.gx + w[3] * P.h.gy) * P.f_h;
  r[0] = P.h.dxp * g_h + w[0] * P.u.dxp + w[1] * P.v.dxp;
  r[1] = P.h.dyp * g_h + w[0] * P.u.dyp + w[1] * P.v.dyp;
  const T qrk = P.q * P.rk;
  const T cs_k = qrk * c * sn;
  r[2] = w[0] * (P.q_k * c * c + qrk * sn * sn) + w[1] * (P.q_k * c * sn - cs_k) +
         w[2] * (P.f_k * c * P.h.gx - P.u.gx) + w[3] * (P.f_k * c * P.h.gy - P.u.gy);
  r[3] = w[0] * (P.q_k * sn * c - cs_k) + w[1] * (P.q_k * sn * sn + qrk * c * c) +
         w[2] * (P.f_k * sn * P.h.gx - P.v.gx) + w[3] * (P.f_k * sn * P.h.gy - P.v.gy);
  // bathymetry nodes of the cell
  {
    const int64_t key = static_cast<int64_t>(P.cb.j) * A.bg.nx + P.cb.i;
    if (key != acc.bkey) {
      flush_bathy(A, acc);
      acc.bkey = key;
    }
    const T fx = P.cb.fx, fy = P.cb.fy;
    const T hxw = w[2] * P.f * A.bg.inv_dx, hyw = w[3] * P.f * A.bg.inv_dy;
    acc.d[0] += g_h * (T(1) - fx) * (T(1) - fy) - hxw - hyw;
    acc.d[1] += g_h * fx * (T(1) - fy) + hxw;
    acc.d[2] += g_h * (T(1) - fx) * fy + hyw;
    acc.d[3] += g_h * fx * fy;
  }
  // current nodes of the cell
  {
    const int64_t key = static_cast<int64_t>(P.cc.j) * A.cg.nx + P.cc.i;
    if (key != acc.ckey) {
      flush_current(A, acc);
      acc.ckey = key;
    }
    const T fx = P.cc.fx, fy = P.cc.fy;
    const T w00 = (T(1) - fx) * (T(1) - fy), w10 = fx * (T(1) - fy), w01 = (T(1) - fx) * fy,
            w11 = fx * fy;
    const T ix = A.cg.inv_dx, iy = A.cg.inv_dy;
    const T kxw2 = s[2] * w[2] * ix, kxw3 = s[2] * w[3] * iy;
    const T kyw2 = s[3] * w[2] * ix, kyw3 = s[3] * w[3] * iy;
    acc.u[0] += w[0] * w00 + kxw2 + kxw3;
    acc.u[1] += w[0] * w10 - kxw2;
    acc.u[2] += w[0] * w01 - kxw3;
    acc.u[3] += w[0] * w11;
    acc.v[0] += w[1] * w00 + kyw2 + kyw3;
    acc.v[1] += w[1] * w10 - kyw2;
    acc.v[2] += w[1] * w01 - kyw3;
    acc.v[3] += w[1] * w11;
  }
}

}  // namespace
}  // namespace mr
