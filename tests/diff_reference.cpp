// The differentiation form's forward, adjoint and tangent-linear passes in
// long double (80 or 128 bits), from the definitions: what the FP64 kernels
// are measured against.  Built by test_gpu_diff_split.py.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

using Q = long double;

struct Grid {
  int64_t nx, ny;
  Q x0, y0, dx, dy;
  Q ix, iy;  // 1 / spacing
};

struct Field {
  const double *a;
  Q v, dx, dy, gx, gy;  // value, surface derivatives, cell differences
};

struct Point {
  int64_t b, c;            // south-west nodes
  Q bx, by, cx, cy;        // fractions
  Field h, u, v;
  Q w, f, qk, qh, fk, fh;  // c_g / k and f, and the partials of c_g and f
  Q c0, s0;                // k / |k|
};

struct Case {
  Grid g, c;
  const double *depth, *u, *v;
  Q dt;
  int64_t steps, n;
};

static bool locate(const Grid &g, Q x, Q y, int64_t *b, Q *fx, Q *fy) {
  const Q i = (x - g.x0) / g.dx, j = (y - g.y0) / g.dy;  // grid lines exactly
  if (!(i >= 0 && j >= 0 && i <= g.nx - 1 && j <= g.ny - 1)) return false;
  const int64_t ci = std::min<int64_t>((int64_t)i, g.nx - 2);
  const int64_t cj = std::min<int64_t>((int64_t)j, g.ny - 2);
  *fx = i - ci;
  *fy = j - cj;
  *b = cj * g.nx + ci;
  return true;
}

static Field take(const double *a, const Grid &g, int64_t b, Q fx, Q fy) {
  const Q v = a[b], ex = (Q)a[b + 1] - v, ey = (Q)a[b + g.nx] - v;
  const Q xy = (Q)a[b + g.nx + 1] - a[b + 1] - a[b + g.nx] + v;
  return Field{a, v + ex * fx + ey * fy + xy * fx * fy, (ex + xy * fy) * g.ix, (ey + xy * fx) * g.iy,
               ex * g.ix, ey * g.iy};
}

static bool eval(const Case &C, const Q *s, Point *p, Q *F) {
  if (!locate(C.g, s[0], s[1], &p->b, &p->bx, &p->by)) return false;
  if (!locate(C.c, s[0], s[1], &p->c, &p->cx, &p->cy)) return false;
  p->h = take(C.depth, C.g, p->b, p->bx, p->by);
  p->u = take(C.u, C.c, p->c, p->cx, p->cy);
  p->v = take(C.v, C.c, p->c, p->cx, p->cy);
  const Q k = sqrtl(s[2] * s[2] + s[3] * s[3]);
  if (!(p->h.v > 0) || !(k > 0)) return false;
  const Q a = k * p->h.v, E = expl(-2 * a), m4 = -expm1l(-4 * a);
  const Q I = 2 * E / m4, coth = (1 + E * E) / m4, N = 2 * a * I, c = 2 * a * coth;
  const Q sg = sqrtl(9.8 * k * tanhl(a));
  p->c0 = s[2] / k;
  p->s0 = s[3] / k;
  p->w = sg * (1 + N) / (2 * k * k);
  p->f = -k * sg * I;
  p->qk = sg / (2 * k * k) * ((N * N - 1) / 2 + N * (1 - c));
  p->qh = sg * I * (1.5L + N / 2 - c);
  p->fk = -p->qh;
  p->fh = sg * k * k * I * (2 * coth - I);
  F[0] = p->w * s[2] + p->u.v;
  F[1] = p->w * s[3] + p->v.v;
  F[2] = p->f * p->h.gx - s[2] * p->u.gx - s[3] * p->v.gx;
  F[3] = p->f * p->h.gy - s[2] * p->u.gy - s[3] * p->v.gy;
  return std::isfinite(F[0]) && std::isfinite(F[1]) && std::isfinite(F[2]) && std::isfinite(F[3]);
}

static void vjp(const Case &C, const Q *s, const Point &p, const Q *w, Q *r, Q *gd, Q *gu, Q *gv) {
  const Q al = w[0] * p.c0 + w[1] * p.s0, ga = w[2] * p.h.gx + w[3] * p.h.gy;
  const Q gh = al * p.qh + ga * p.fh, ak = (p.qk - p.w) * al + p.fk * ga;
  r[0] = gh * p.h.dx + w[0] * p.u.dx + w[1] * p.v.dx;
  r[1] = gh * p.h.dy + w[0] * p.u.dy + w[1] * p.v.dy;
  r[2] = p.w * w[0] + ak * p.c0 - w[2] * p.u.gx - w[3] * p.u.gy;
  r[3] = p.w * w[1] + ak * p.s0 - w[2] * p.v.gx - w[3] * p.v.gy;
  auto add = [](Q *g, int64_t nx, Q val, Q fx, Q fy, Q x, Q y) {
    g[0] += val * (1 - fx) * (1 - fy) - x - y;
    g[1] += val * fx * (1 - fy) + x;
    g[nx] += val * (1 - fx) * fy + y;
    g[nx + 1] += val * fx * fy;
  };
  add(gd + p.b, C.g.nx, gh, p.bx, p.by, w[2] * p.f * C.g.ix, w[3] * p.f * C.g.iy);
  add(gu + p.c, C.c.nx, w[0], p.cx, p.cy, -s[2] * w[2] * C.c.ix, -s[2] * w[3] * C.c.iy);
  add(gv + p.c, C.c.nx, w[1], p.cx, p.cy, -s[3] * w[2] * C.c.ix, -s[3] * w[3] * C.c.iy);
}

static Case make(const int64_t *nodes, const double *geom, const double *depth, const double *u,
                 const double *v, double dt, int64_t steps, int64_t n) {
  auto inv = [](Q d) { return 1 / d; };
  return Case{Grid{nodes[0], nodes[1], geom[0], geom[1], geom[2], geom[3], inv(geom[2]), inv(geom[3])},
              Grid{nodes[2], nodes[3], geom[4], geom[5], geom[6], geom[7],
                   inv(geom[6]), inv(geom[7])},
              depth, u, v, dt, steps, n};
}

// nodes: (nx, ny) of both grids; geom: (x0, y0, dx, dy) of both; rays, end,
// grad_end, g0: [4][n]; rays first..last-1.
extern "C" void adjoint(const int64_t *nodes, const double *geom, const double *depth,
                        const double *u, const double *v, double dt, int64_t steps, int64_t n,
                        int64_t first, int64_t last, const double *rays, const double *grad_end,
                        double *end, uint8_t *status, double *g0, double *gd, double *gu,
                        double *gv) {
  const Case C = make(nodes, geom, depth, u, v, dt, steps, n);
  std::vector<Q> Y(16 * steps + 4), D(C.g.nx * C.g.ny), U(C.c.nx * C.c.ny), V(U.size());
  for (int64_t r = first; r < last; ++r) {
    Q y[4], F[4], sum[4];
    Point p;
    bool ok = true;
    for (int q = 0; q < 4; ++q) y[q] = rays[q * n + r];
    for (int64_t s = 0; s < steps && ok; ++s) {
      Q *R = &Y[16 * s];
      for (int st = 0; st < 4 && ok; ++st) {
        for (int q = 0; q < 4; ++q)
          R[4 * st + q] = st == 0 ? y[q] : y[q] + F[q] * (st == 3 ? C.dt : C.dt / 2);
        ok = eval(C, R + 4 * st, &p, F);
        for (int q = 0; q < 4; ++q)
          sum[q] = (st == 0 ? 0 : sum[q]) + F[q] * (st == 0 || st == 3 ? 1 : 2);
      }
      for (int q = 0; q < 4; ++q) y[q] += sum[q] * C.dt / 6;
    }
    status[r] = !ok;
    for (int q = 0; q < 4; ++q) {
      end[q * n + r] = ok ? (double)y[q] : NAN;
      g0[q * n + r] = 0.0;
    }
    if (!ok) continue;
    Q lam[4];
    for (int q = 0; q < 4; ++q) lam[q] = grad_end[q * n + r];
    for (int64_t s = steps - 1; s >= 0; --s) {
      Q rr[4] = {0, 0, 0, 0}, tot[4] = {0, 0, 0, 0}, w[4];
      for (int st = 3; st >= 0; --st) {
        const Q c = C.dt / (st == 0 || st == 3 ? 6 : 3), f = st == 3 ? 0 : st == 2 ? C.dt : C.dt / 2;
        for (int q = 0; q < 4; ++q) w[q] = lam[q] * c + f * rr[q];
        eval(C, &Y[16 * s + 4 * st], &p, F);
        vjp(C, &Y[16 * s + 4 * st], p, w, rr, D.data(), U.data(), V.data());
        for (int q = 0; q < 4; ++q) tot[q] += rr[q];
      }
      for (int q = 0; q < 4; ++q) lam[q] += tot[q];
    }
    for (int q = 0; q < 4; ++q) g0[q * n + r] = (double)lam[q];
  }
  for (size_t i = 0; i < D.size(); ++i) gd[i] = (double)D[i];
  for (size_t i = 0; i < U.size(); ++i) {
    gu[i] = (double)U[i];
    gv[i] = (double)V[i];
  }
}

static void jvp(const Case &C, const Q *s, const Point &p, const Q *ds, const double *dd,
                const double *du, const double *dv, Q *dF) {
  Field d{}, u{}, v{};
  if (dd) d = take(dd, C.g, p.b, p.bx, p.by);
  if (du) u = take(du, C.c, p.c, p.cx, p.cy);
  if (dv) v = take(dv, C.c, p.c, p.cx, p.cy);
  const Q dh = p.h.dx * ds[0] + p.h.dy * ds[1] + d.v, dk = p.c0 * ds[2] + p.s0 * ds[3];
  const Q k = p.c0 * s[2] + p.s0 * s[3], dw = (p.qk - p.w) / k * dk + p.qh / k * dh;
  const Q df = p.fk * dk + p.fh * dh;
  dF[0] = p.w * ds[2] + s[2] * dw + p.u.dx * ds[0] + p.u.dy * ds[1] + u.v;
  dF[1] = p.w * ds[3] + s[3] * dw + p.v.dx * ds[0] + p.v.dy * ds[1] + v.v;
  dF[2] = df * p.h.gx + p.f * d.gx - ds[2] * p.u.gx - s[2] * u.gx - ds[3] * p.v.gx - s[3] * v.gx;
  dF[3] = df * p.h.gy + p.f * d.gy - ds[2] * p.u.gy - s[2] * u.gy - ds[3] * p.v.gy - s[3] * v.gy;
}

// dd, du, dv: tangent fields or null; dstate, d_end: [4][n].
extern "C" void tangent(const int64_t *nodes, const double *geom, const double *depth,
                        const double *u, const double *v, double dt, int64_t steps, int64_t n,
                        int64_t first, int64_t last, const double *rays, const double *dstate,
                        const double *dd, const double *du, const double *dv, double *end,
                        uint8_t *status, double *d_end) {
  const Case C = make(nodes, geom, depth, u, v, dt, steps, n);
  for (int64_t r = first; r < last; ++r) {
    Q y[4], dy[4], F[4], dF[4], t[4], d[4], sum[4], dsum[4];
    Point p;
    bool ok = true;
    for (int q = 0; q < 4; ++q) {
      y[q] = rays[q * n + r];
      dy[q] = dstate[q * n + r];
    }
    for (int64_t s = 0; s < steps && ok; ++s) {
      for (int st = 0; st < 4 && ok; ++st) {
        for (int q = 0; q < 4; ++q) {
          const Q h = st == 3 ? C.dt : C.dt / 2;
          t[q] = st == 0 ? y[q] : y[q] + F[q] * h;
          d[q] = st == 0 ? dy[q] : dy[q] + dF[q] * h;
        }
        ok = eval(C, t, &p, F);
        if (ok) jvp(C, t, p, d, dd, du, dv, dF);
        for (int q = 0; q < 4; ++q) {
          const Q wt = st == 0 || st == 3 ? 1 : 2;
          sum[q] = (st == 0 ? 0 : sum[q]) + wt * F[q];
          dsum[q] = (st == 0 ? 0 : dsum[q]) + wt * dF[q];
        }
      }
      for (int q = 0; q < 4; ++q) {
        y[q] += sum[q] * C.dt / 6;
        dy[q] += dsum[q] * C.dt / 6;
      }
    }
    status[r] = !ok;
    for (int q = 0; q < 4; ++q) {
      end[q * n + r] = ok ? (double)y[q] : NAN;
      d_end[q * n + r] = ok ? (double)dy[q] : NAN;
    }
  }
}
