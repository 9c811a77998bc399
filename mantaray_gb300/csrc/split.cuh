// split.cuh -- the ray equations on pairs of floats, with one FP64 anchor a
// step, for the plain integrator on gridded bathymetry (rk4_f64_grid.cu).
//
// GB300 issues 2 FP64 lanes per SM and clock against 128 FP32 lanes, so an
// FP64 operation costs 64 FP32 ones.  A value held as an unevaluated sum of
// two floats (high + low, about 48 bits) takes 4-12 FP32 operations per
// operation (Dekker 1971; Knuth's two-sum; products by FMA).  48 bits are not
// 53, so a step's derivative is not taken from the pairs alone:
//
//   x' = x + dt A + (dt/6) D,   D = 2 (d2 - d1) + 2 (d3 - d1) + (d4 - d1),
//
// where A is the position derivative of the first stage in FP64 and d1..d4
// the four stages' derivatives in pairs.  The stages of one step differ by
// 1e-2 to 1e-4 of the derivative, so the pairs' error enters D at 2^-55 to
// 2^-60 of the step, below the rounding of x' itself, and where the stages
// do not differ (deep water, uniform current) D is exactly zero.  The
// wavenumber's derivative is a small fraction of the wavenumber per step, so
// its increment is taken from the pairs directly.
//
// Domain (split_ok): depth 2^-7..2^17 m, k^2 2^-40..2^40, |u| < 2^20 and cell
// gradients below 2^20.  Everything else, NaN and infinities included, is
// left to the FP64 form (ray_exact.cuh).
//
// What is the same for x and y runs on packed instructions (packed.cuh), which
// the assembler contracts: every product there that meets a sum is exact (by a
// power of two or -1), in a written FMA, or two scalar products (vmul_rn: the
// same bits as packed ones today, at 0 to 1.3% of the time).
//
// Host and device code: the host build is what the CPU tests check against
// 64-bit and wider arithmetic.  -fmad=false / -ffp-contract=off: every fused
// operation is written as one.
#pragma once

#include <math.h>
#include <stdint.h>

#include "bits.h"
#include "exp_table.h"
#include "packed.cuh"

namespace mr {
// The two forms of the pairs' products have names of their own, so that units
// of both can be linked.
#ifdef MR_SPLIT_LOW_PRODUCT
inline namespace pairs_low_product {
#else
inline namespace pairs {
#endif
using ::mr::both;

// Functions that read the tables: device code where there is a device.
#if defined(__CUDACC__)
#define MR_SPLIT __device__ __forceinline__
#else
#define MR_SPLIT inline
#endif

struct F2 { float h, l; };  // the value h + l, l a few ulps of h at most

MR_HD float fma32(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return fmaf(a, b, c);
#endif
}
// First guesses of 1/sqrt(x) and 1/x, good to about 2^-22; refined below.  The
// host's are given errors of that size.
MR_HD float guess_error(float r) {
  return r * (1.0f + (static_cast<float>(bits_of(r) * 2654435761u >> 24) - 127.5f) * 0x1p-29f);
}
MR_HD float rsqrt_guess(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return guess_error(1.0f / sqrtf(x));
#endif
}
MR_HD float rcp_guess(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return guess_error(1.0f / x);
#endif
}

// s + e = a + b exactly; fast: |a| >= |b| or a = 0.
MR_HD F2 two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return F2{s, (a - (s - bb)) + (b - bb)};
}
MR_HD F2 fast_two_sum(float a, float b) {
  const float s = a + b;
  return F2{s, b - (s - a)};
}
MR_HD F2 neg(F2 a) { return F2{-a.h, -a.l}; }
MR_HD F2 scale(float p2, F2 a) { return F2{p2 * a.h, p2 * a.l}; }  // p2: a power of two
// Sums and products leave their low half unrounded into the high one (|l| up
// to a few ulps of h): the operations below lose a.l b.l only, 2^-45 of the
// product, and the rounding steps saved are a third of the instructions and
// of the dependent chain.  MR_SPLIT_LOW_PRODUCT keeps a.l b.l, for a unit
// whose results carry products' errors on (diff_split.cu; the trajectories
// gain nothing from it).
MR_HD F2 add(F2 a, F2 b) {
  const F2 s = two_sum(a.h, b.h);
  return F2{s.h, s.l + (a.l + b.l)};
}
MR_HD F2 add_f(F2 a, float b) {
  const F2 s = two_sum(a.h, b);
  return F2{s.h, s.l + a.l};
}
// a + b, both positive: the larger first.
MR_HD F2 add_pos(F2 a, F2 b) {
  const bool swap = b.h > a.h;
  const F2 s = fast_two_sum(swap ? b.h : a.h, swap ? a.h : b.h);
  return F2{s.h, s.l + (a.l + b.l)};
}
// a + b where |a| >= |b|.
MR_HD F2 add_small(F2 a, F2 b) {
  const F2 s = fast_two_sum(a.h, b.h);
  return F2{s.h, s.l + (a.l + b.l)};
}
MR_HD F2 mul(F2 a, F2 b) {
  const float p = a.h * b.h;
#ifdef MR_SPLIT_LOW_PRODUCT
  return F2{p, fma32(a.h, b.h, -p) + fma32(a.h, b.l, fma32(a.l, b.l, a.l * b.h))};
#else
  return F2{p, fma32(a.h, b.h, -p) + fma32(a.h, b.l, a.l * b.h)};
#endif
}
MR_HD F2 mul_f(F2 a, float b) {
  const float p = a.h * b;
  return F2{p, fma32(a.l, b, fma32(a.h, b, -p))};
}
MR_HD F2 sqr(F2 a) {
  const float p = a.h * a.h;
#ifdef MR_SPLIT_LOW_PRODUCT
  return F2{p, fma32(a.h + a.h, a.l, fma32(a.l, a.l, fma32(a.h, a.h, -p)))};
#else
  return F2{p, fma32(a.h + a.h, a.l, fma32(a.h, a.h, -p))};
#endif
}
// 1/sqrt(x), one Newton step of third order on the guess: e = 1 - x r^2.
MR_HD F2 rsqrt2(F2 x) {
  const float r = rsqrt_guess(x.h);
  const float p = r * r;
  const float pe = fma32(r, r, -p);
  const float e = fma32(-x.h, p, 1.0f) - fma32(x.h, pe, x.l * p);
  return fast_two_sum(r, r * (e * fma32(0.375f, e, 0.5f)));
}
MR_HD F2 rcp2(F2 x) {
  const float r = rcp_guess(x.h);
  const float e = fma32(-x.l, r, fma32(-x.h, r, 1.0f));
  return fast_two_sum(r, r * fma32(e, e, e));
}

// ---------------------------------------------- two lanes at once (x, y) --

struct V2 { V h, l; };  // a pair (F2) for each of x and y

MR_HD V2 both(F2 a) { return V2{both(a.h), both(a.l)}; }
MR_HD F2 x_of(V2 a) { return F2{a.h.x, a.l.x}; }
MR_HD F2 y_of(V2 a) { return F2{a.h.y, a.l.y}; }
MR_HD V2 zero2() { return V2{both(0.0f), both(0.0f)}; }

MR_HD V2 two_sum(V a, V b) {
  const V s = vadd(a, b);
  const V bb = vsub(s, a);
  return V2{s, vadd(vsub(a, vsub(s, bb)), vsub(b, bb))};
}
MR_HD V2 add(V2 a, V2 b) {
  const V2 s = two_sum(a.h, b.h);
  return V2{s.h, vadd(s.l, vadd(a.l, b.l))};
}
MR_HD V2 add_f(V2 a, V b) {
  const V2 s = two_sum(a.h, b);
  return V2{s.h, vadd(s.l, a.l)};
}
MR_HD V2 sub(V2 a, V2 b) {
  const V s = vsub(a.h, b.h);
  const V bb = vsub(s, a.h);  // -(the part of b that s holds)
  const V e = vsub(vsub(a.h, vsub(s, bb)), vadd(b.h, bb));
  return V2{s, vadd(e, vsub(a.l, b.l))};
}
MR_HD V2 mul(V2 a, V2 b) {
  const V p = vmul_rn(a.h, b.h);
  const V e = vfma(a.h, b.h, vmul(p, both(-1.0f)));
#ifdef MR_SPLIT_LOW_PRODUCT
  return V2{p, vfma(a.l, b.h, vfma(a.h, b.l, vfma(a.l, b.l, e)))};
#else
  return V2{p, vfma(a.l, b.h, vfma(a.h, b.l, e))};
#endif
}
MR_HD V2 mul_f(V2 a, V b) {
  const V p = vmul_rn(a.h, b);
  return V2{p, vfma(a.l, b, vfma(a.h, b, vmul(p, both(-1.0f))))};
}
MR_HD V2 scale(float p2, V2 a) { return V2{vmul(a.h, both(p2)), vmul(a.l, both(p2))}; }
// a.x^2 + a.y^2
MR_HD F2 norm2(V2 a) {
  const V p = vmul_rn(a.h, a.h);
  const V e = vfma(vadd(a.h, a.h), a.l, vfma(a.h, a.h, vmul(p, both(-1.0f))));
  return add_pos(F2{p.x, e.x}, F2{p.y, e.y});
}

// ------------------------------------------------------ doubles and pairs --
// The conversions are integer operations (the conversion instructions run on
// the FP64 pipe).

// f as a double; a zero or subnormal f reads as up to +-2^-126.
MR_HD double f2d_normal(float f) {
  const uint32_t u = bits_of(f);
  return double_of((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u), u << 29);
}
MR_HD double f2d_zero(float f) { return f == 0.0f ? 0.0 : f2d_normal(f); }
// Either half may be 0 (a difference can be all low half).
MR_HD double to_double(F2 a) { return f2d_zero(a.h) + f2d_zero(a.l); }
// v = h + m + r exactly: the top 24 bits, the next 23 and the last 6 (for
// magnitudes outside 2^-73..2^126, zero among them, h = (float)v alone).
MR_HD void split3(double v, float *h, float *m, float *r) {
  const uint64_t b = bits_of(v);
  const uint32_t hi = static_cast<uint32_t>(b >> 32), lo = static_cast<uint32_t>(b);
  const uint32_t e = (hi >> 20) & 0x7ffu;
  if (e - 950u < 200u) {
    *h = float_of((hi & 0x80000000u) | ((e - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29));
    const float s = float_of((hi & 0x80000000u) | ((e - 948u) << 23));  // 2^(e - 52), signed
    const uint32_t n = lo & 0x1fffffffu;
    *m = (float_of(0x4b000000u | (n >> 6)) - 8388608.0f) * (64.0f * s);
    *r = (float_of(0x4b000000u | (n & 63u)) - 8388608.0f) * s;
  } else {
    *h = d2f(v);
    *m = *r = 0.0f;
  }
}
MR_HD F2 to_pair(double v) {
  F2 a;
  float r;
  split3(v, &a.h, &a.l, &r);
  a.l += r;
  return a;
}
// v / 2 and v / 4 for normal v well inside the exponent range.
MR_HD double half_of(double v) {
  const uint64_t b = bits_of(v);
  return double_of(static_cast<uint32_t>(b >> 32) - 0x100000u, static_cast<uint32_t>(b));
}
MR_HD double quarter_of(double v) {
  const uint64_t b = bits_of(v);
  return double_of(static_cast<uint32_t>(b >> 32) - 0x200000u, static_cast<uint32_t>(b));
}

// ------------------------------------------------------- the derivatives --

// The fields at a point: depth and its cell gradient, current, and the
// current's cell gradients (du/dx, du/dy) and (dv/dx, dv/dy).
struct Sample {
  float h;
  V g;
  V2 uv, du, dv;
};

// Whether the pairs cover a point (NaN fails every comparison).
MR_HD bool split_ok(const Sample &s, float k2) {
  return s.h > 0.0078125f && s.h < 131072.0f && fabsf(s.uv.h.x) < 1048576.0f &&
         fabsf(s.uv.h.y) < 1048576.0f && k2 > 0x1p-40f && k2 < 0x1p40f;
}

// exp(-2a) = q and m = 1 - q from x = -2a in (-44.5, 0]: with
// n = round(-x 256 / ln 2), x = -n ln2/256 + r, |r| <= ln2/512, q =
// 2^(-n/256) (1 + p), p = e^r - 1 (Tang 1989).  For n < 256 the table's own
// 1 - 2^(-n/256) keeps m relatively accurate as it tends to 0.
MR_SPLIT void split_exp(F2 x, int *n_out, F2 *q, F2 *m) {
  const float nf = rintf(x.h * -369.3299304675746f);
  const int n = static_cast<int>(nf);
  // r = x + n ln2/256 in three parts (10 bits: exact product; 24; the rest)
  const float r1 = fma32(nf, 0x1.628p-9f, x.h);
  const float p2 = nf * 0x1.90bfbep-19f;
  const float p2e = fma32(nf, 0x1.90bfbep-19f, -p2);
  const F2 s = two_sum(r1, p2);
  const F2 r = fast_two_sum(s.h, s.l + (x.l + fma32(nf, 0x1.1cf79ap-44f, p2e)));
  // p = r + r^2/2 + r^3/6 + r^4/24; r^3/6 is below 5e-10
  const float r2 = r.h * r.h;
  const float r2e = fma32(r.h, r.h, -r2);
  float tail = r2 * r.h * fma32(r.h, 1.0f / 24.0f, 1.0f / 6.0f);
  tail = fma32(0.5f, r2e, tail);
  tail = fma32(r.h, r.l, tail);
  const F2 ps = fast_two_sum(r.h, 0.5f * r2);
  const F2 p = F2{ps.h, ps.l + (r.l + tail)};
#if defined(__CUDA_ARCH__)
  const float4 t = __ldg(reinterpret_cast<const float4 *>(kExp32) + (n & 255));
  const float th = t.x, tl = t.y, uh = t.z, ul = t.w;
#else
  const float th = kExp32[n & 255].th, tl = kExp32[n & 255].tl, uh = kExp32[n & 255].uh,
              ul = kExp32[n & 255].ul;
#endif
  const float sc = float_of(static_cast<uint32_t>(127 - (n >> 8)) << 23);
  const F2 T = F2{th * sc, tl * sc};
  F2 U = F2{uh, ul};
  if (n >= 256) {
    const F2 one = fast_two_sum(1.0f, -T.h);
    U = F2{one.h, one.l - T.l};
  }
  const F2 tp = mul(T, p);
  *q = add_small(T, tp);
  *m = add(U, neg(tp));
  *n_out = n;
}

// exp(-2a) = q and m = 1 - q in FP64, n as split_exp finds it (8 FP64
// operations, the table as there).
MR_SPLIT void anchor_exp(double a, int n, double *q, double *m) {
  // r/2 = -a + (n/2) ln2/256, the halves exact
  const double nh = f2d_zero(0.5f * static_cast<float>(n));
  const double rh = fma(nh, 0x1.cf79abc9e3b3ap-48, fma(nh, 0x1.62e42fefap-9, -a));
  // p = e^r - 1 = r + 2 (r/2)^2 + r^3/6 + ..., the tail in FP32 (r^3/6 is
  // below 5e-10)
  const float rf = 2.0f * d2f(rh);
  const float tail = rf * rf * rf * fma32(rf, fma32(rf, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f);
  const double rr = rh + rh;
  const double p = fma(rr, rh, rr) + f2d(tail);
#if defined(__CUDA_ARCH__)
  const double2 tu = __ldg(reinterpret_cast<const double2 *>(kExp64) + (n & 255));
  double T = tu.x, U = tu.y;
#else
  double T = kExp64[n & 255].t, U = kExp64[n & 255].u;
#endif
  if (n >= 256) {
    const uint64_t tb = bits_of(T);
    T = double_of(static_cast<uint32_t>(tb >> 32) - (static_cast<uint32_t>(n >> 8) << 20),
                  static_cast<uint32_t>(tb));
    U = 1.0 - T;
  }
  *m = fma(-T, p, U);
  *q = fma(T, p, T);
}

// A wavenumber with its square, inverse and magnitude.  Apart from split_rhs
// so that a stage can compute them beside its position, before its lookup.
struct Wave {
  V2 kv;
  F2 k2, rk, k;
};
MR_HD Wave wave_of(V2 kv) {
  Wave w;
  w.kv = kv;
  w.k2 = norm2(kv);
  w.rk = rsqrt2(w.k2);
  w.k = mul(w.k2, w.rk);
  return w;
}

// The derivatives (dx, dy) in d and (dkx, dky) in dk at a wavenumber, in
// pairs.  With a = kh, q = exp(-2a), m = 1 - q, z = 1/(1 + q), rho =
// 1/sqrt(k m (1 + q)):
//   c_g / k = sqrt(g)/2 rho (m + 4 a q z) / k,
//   refraction factor f = -2 sqrt(g) k^2 q z rho,
// which are the reference's group velocity and -k/2 sqrt(g k tanh a) /
// (sinh a cosh a).  Beyond a = 22, q is below half an ulp of 1 and the
// deep-water forms are exact: c_g / k = sqrt(g)/2 k2^(-3/4), f = 0.
//
// ANCHOR: also c_g / k in FP64 at (kx, ky), to *speed.  1/k, 1/(1 + q) and
// 1/sqrt(k m (1 + q)) (deep water: k2^(-3/4)) start from the pairs and take
// one Newton correction, exp(-2a) comes from the FP64 table, so its error is
// FP64 rounding: 33 FP64 operations (10 in deep water), with no division,
// expm1 or rsqrt.
template <bool ANCHOR>
MR_SPLIT void split_rhs(const Sample &s, const Wave &wv, V2 *d, V2 *dk, double kx, double ky,
                        double *speed) {
  constexpr double kHalfSqrtG = 0x1.90b410d07f01ep+0;    // sqrt(9.8) / 2
  const F2 kC = F2{0x1.90b41p+0f, 0x1.a0fe04p-25f};      // the same as a pair
  const V2 kv = wv.kv;
  const F2 k2 = wv.k2, rk = wv.rk, k = wv.k;
  const F2 a = mul_f(k, s.h);
  const V2 t = add(mul(both(F2{kv.h.x, kv.l.x}), s.du), mul(both(F2{kv.h.y, kv.l.y}), s.dv));
  const double k2d = ANCHOR ? fma(kx, kx, ky * ky) : 0.0;
  F2 w;
  if (a.h > 22.0f) {
    const F2 w0 = mul(rk, rsqrt2(k));
    w = mul(kC, w0);
    *dk = zero2();
    if (ANCHOR) {
      const double wd = f2d_normal(w0.h) + f2d_normal(w0.l);
      const double w2 = wd * wd;
      const double e = fma(-quarter_of(w2 * w2), k2d * k2d * k2d, 0.25);
      *speed = kHalfSqrtG * fma(wd, e, wd);
    }
  } else {
    int n;
    F2 q, m;
    split_exp(scale(-2.0f, a), &n, &q, &m);
    const F2 onep = fast_two_sum(1.0f, q.h);
    const F2 q1 = F2{onep.h, onep.l + q.l};
    const F2 z = rcp2(q1);
    const F2 rho = rsqrt2(mul(mul(k, m), q1));
    const F2 qz = mul(q, z);
    const F2 b = add(m, scale(4.0f, mul(a, qz)));
    const F2 cr = mul(kC, rho);
    w = mul(mul(cr, b), rk);
    const F2 f = mul(mul(scale(-4.0f, cr), k2), qz);
    *dk = mul_f(both(f), s.g);
    if (ANCHOR) {
      const double rk0 = f2d_normal(rk.h) + f2d_normal(rk.l);
      const double k0 = k2d * rk0;
      const double ek = fma(-half_of(k0), rk0, 0.5);
      const double kd = fma(k0, ek, k0);
      const double rkd = fma(rk0, ek, rk0);
      const double ad = kd * f2d_normal(s.h);
      double qd, md;
      anchor_exp(ad, n, &qd, &md);
      const double q1d = 1.0 + qd;
      const double z0 = f2d_normal(z.h) + f2d_normal(z.l);
      const double zd = fma(z0, fma(-q1d, z0, 1.0), z0);
      const double D = kd * md * q1d;
      const double r0 = f2d_normal(rho.h) + f2d_normal(rho.l);
      const double er = fma(-half_of(D * r0), r0, 0.5);
      const double rhod = fma(r0, er, r0);
      *speed = kHalfSqrtG * rhod * fma(4.0 * ad, qd * zd, md) * rkd;
    }
  }
  *d = add(mul(both(w), kv), s.uv);
  *dk = sub(*dk, t);
}

}  // inline namespace
}  // namespace mr
