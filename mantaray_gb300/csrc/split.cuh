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
// Host and device code: the host build is what the CPU tests check against
// 64-bit and wider arithmetic.  -fmad=false / -ffp-contract=off: every fused
// operation is written as one.
#pragma once

#include <math.h>
#include <stdint.h>

#include "bits.h"
#include "exp_table.h"

namespace mr {

// Functions that read the tables: device code where there is a device.
#if defined(__CUDACC__)
#define MR_SPLIT __device__ __forceinline__
#else
#define MR_SPLIT inline
#endif

struct F2 { float h, l; };  // the value h + l, |l| <= ulp(h)/2

MR_HD float fma32(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return fmaf(a, b, c);
#endif
}
// First guesses of 1/sqrt(x) and 1/x, good to about 2^-22; refined below.
MR_HD float rsqrt_guess(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / sqrtf(x);
#endif
}
MR_HD float rcp_guess(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
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
MR_HD F2 twice(F2 a) { return F2{2.0f * a.h, 2.0f * a.l}; }
MR_HD F2 add(F2 a, F2 b) {
  const F2 s = two_sum(a.h, b.h);
  return fast_two_sum(s.h, s.l + (a.l + b.l));
}
MR_HD F2 add_f(F2 a, float b) {
  const F2 s = two_sum(a.h, b);
  return fast_two_sum(s.h, s.l + a.l);
}
// a + b, both positive: the larger first.
MR_HD F2 add_pos(F2 a, F2 b) {
  const bool swap = b.h > a.h;
  const F2 s = fast_two_sum(swap ? b.h : a.h, swap ? a.h : b.h);
  return fast_two_sum(s.h, s.l + (a.l + b.l));
}
// a + b where |a| >= |b|.
MR_HD F2 add_small(F2 a, F2 b) {
  const F2 s = fast_two_sum(a.h, b.h);
  return fast_two_sum(s.h, s.l + (a.l + b.l));
}
MR_HD F2 mul(F2 a, F2 b) {
  const float p = a.h * b.h;
  float e = fma32(a.h, b.h, -p);
  e = fma32(a.h, b.l, e);
  e = fma32(a.l, b.h, e);
  return fast_two_sum(p, e);
}
MR_HD F2 mul_f(F2 a, float b) {
  const float p = a.h * b;
  const float e = fma32(a.l, b, fma32(a.h, b, -p));
  return fast_two_sum(p, e);
}
MR_HD F2 sqr(F2 a) {
  const float p = a.h * a.h;
  const float e = fma32(a.h + a.h, a.l, fma32(a.h, a.h, -p));
  return fast_two_sum(p, e);
}
// 1/sqrt(x), one Newton step of third order on the guess: e = 1 - x r^2.
MR_HD F2 rsqrt2(F2 x) {
  const float r = rsqrt_guess(x.h);
  const float p = r * r;
  const float pe = fma32(r, r, -p);
  float e = fma32(-x.h, p, 1.0f);
  e = fma32(-x.h, pe, e);
  e = fma32(-x.l, p, e);
  return fast_two_sum(r, r * (e * fma32(0.375f, e, 0.5f)));
}
MR_HD F2 rcp2(F2 x) {
  const float r = rcp_guess(x.h);
  float e = fma32(-x.h, r, 1.0f);
  e = fma32(-x.l, r, e);
  return fast_two_sum(r, r * fma32(e, e, e));
}

// Doubles and pairs.  The conversions are integer operations (the conversion
// instructions run on the FP64 pipe); to_double adds the two halves there.
MR_HD double f2d_normal(float f) {
  const uint32_t u = bits_of(f);
  return double_of((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u), u << 29);
}
// a.h = 0 gives 0 (a.l is 0 there); a subnormal or zero a.l reads as
// +-2^-127, which the sum rounds away unless a.h is below 2^-74.
MR_HD double to_double(F2 a) {
  const double s = f2d_normal(a.h) + f2d_normal(a.l);
  return a.h == 0.0f ? 0.0 : s;
}
MR_HD F2 to_pair(double v) {
  const float h = d2f(v);
  return F2{h, d2f(v - f2d(h))};
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

// The fields at a point: depth and its cell gradient, current, and the
// current's cell gradients.
struct Sample {
  float h, gx, gy;
  F2 u, v;
  F2 ux, uy, vx, vy;
};

// Whether the pairs cover a point (NaN fails every comparison).
MR_HD bool split_ok(const Sample &s, float k2) {
  return s.h > 0.0078125f && s.h < 131072.0f && s.u.h > -1048576.0f && s.u.h < 1048576.0f &&
         s.v.h > -1048576.0f && s.v.h < 1048576.0f && k2 > 0x1p-40f && k2 < 0x1p40f;
}

// What the first stage hands to the FP64 anchor: the same quantities to
// about 2^-46, which one FP64 correction each makes exact to FP64 rounding.
struct Anchor {
  bool deep;
  int n;           // exp(-2kh) = 2^(-n/256) exp(r)
  F2 rk, rho, z;   // 1/k, 1/sqrt(k m (1 + q)), 1/(1 + q)
  F2 w;            // deep water: k2^(-3/4)
};

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
  const F2 p = fast_two_sum(ps.h, ps.l + (r.l + tail));
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
    U = fast_two_sum(one.h, one.l - T.l);
  }
  const F2 tp = mul(T, p);
  *q = add_small(T, tp);
  *m = add(U, neg(tp));
  *n_out = n;
}

// The derivatives (dx, dy, dkx, dky) at wavenumber (kx, ky), in pairs, and
// the anchor's quantities when ANCHOR.  With a = kh, q = exp(-2a), m = 1 - q,
// z = 1/(1 + q), rho = 1/sqrt(k m (1 + q)):
//   c_g / k = sqrt(g)/2 rho (m + 4 a q z) / k,
//   refraction factor f = -2 sqrt(g) k^2 q z rho,
// which are the reference's group velocity and -k/2 sqrt(g k tanh a) /
// (sinh a cosh a).  Beyond a = 22, q is below half an ulp of 1 and the
// deep-water forms are exact: c_g / k = sqrt(g)/2 k2^(-3/4), f = 0.
template <bool ANCHOR>
MR_SPLIT void split_rhs(const Sample &s, F2 kx, F2 ky, F2 k2, F2 d[4], Anchor *an) {
  const F2 rk = rsqrt2(k2);
  const F2 k = mul(k2, rk);
  const F2 a = mul_f(k, s.h);
  const F2 kC = F2{0x1.90b41p+0f, 0x1.a0fe04p-25f};      // sqrt(9.8) / 2
  F2 w, f = F2{0.0f, 0.0f};
  const bool deep = a.h > 22.0f;
  if (deep) {
    const F2 w0 = mul(rk, rsqrt2(k));
    w = mul(kC, w0);
    if (ANCHOR) {
      an->w = w0;
      an->n = 0;
      an->rk = an->rho = an->z = w0;
    }
  } else {
    int n;
    F2 q, m;
    split_exp(F2{-2.0f * a.h, -2.0f * a.l}, &n, &q, &m);
    const F2 onep = fast_two_sum(1.0f, q.h);
    const F2 q1 = fast_two_sum(onep.h, onep.l + q.l);
    const F2 z = rcp2(q1);
    const F2 rho = rsqrt2(mul(mul(k, m), q1));
    const F2 qz = mul(q, z);
    const F2 aqz = mul(a, qz);
    const F2 b = add(m, F2{4.0f * aqz.h, 4.0f * aqz.l});
    const F2 cr = mul(kC, rho);
    w = mul(mul(cr, b), rk);
    const F2 c4 = F2{-4.0f * cr.h, -4.0f * cr.l};        // -2 sqrt(9.8) rho
    f = mul(mul(c4, k2), qz);
    if (ANCHOR) {
      an->rk = rk;
      an->rho = rho;
      an->z = z;
      an->n = n;
      an->w = w;
    }
  }
  if (ANCHOR) an->deep = deep;
  d[0] = add(mul(w, kx), s.u);
  d[1] = add(mul(w, ky), s.v);
  const F2 t2 = add(mul(kx, s.ux), mul(ky, s.vx));
  const F2 t3 = add(mul(kx, s.uy), mul(ky, s.vy));
  if (deep) {
    d[2] = neg(t2);
    d[3] = neg(t3);
  } else {
    d[2] = add(mul_f(f, s.gx), neg(t2));
    d[3] = add(mul_f(f, s.gy), neg(t3));
  }
}

// c_g / k in FP64 at (kx, ky) and depth h: each of 1/k, exp(-2a), 1/(1 + q)
// and 1/sqrt(k m (1 + q)) (deep water: k2^(-3/4)) starts from the pair of
// split_rhs and takes one Newton correction, so its error is FP64 rounding.
// 33 FP64 operations (10 in deep water), with no division, expm1 or rsqrt of
// its own.
MR_SPLIT double anchor_speed(const Anchor &an, double kx, double ky, float h) {
  constexpr double kHalfSqrtG = 0x1.90b410d07f01ep+0;    // sqrt(9.8) / 2
  const double k2 = fma(kx, kx, ky * ky);
  if (an.deep) {
    const double w0 = f2d_normal(an.w.h) + f2d_normal(an.w.l);
    const double w2 = w0 * w0;
    const double e = fma(-quarter_of(w2 * w2), k2 * k2 * k2, 0.25);
    return kHalfSqrtG * fma(w0, e, w0);
  }
  const double rk0 = f2d_normal(an.rk.h) + f2d_normal(an.rk.l);
  const double t = k2 * rk0;
  const double ek = fma(-half_of(t), rk0, 0.5);
  const double k = fma(t, ek, t);
  const double rk = fma(rk0, ek, rk0);
  const double a = k * f2d_normal(h);
  // r = -2a + n ln2/256; half of it, exactly scaled
  const float nf = static_cast<float>(an.n);
  const double nh = half_of(f2d(nf + 0.0f));
  const double rh0 = an.n == 0 ? -a : fma(nh, 0x1.62e42fefap-9, -a);
  const double rh = an.n == 0 ? rh0 : fma(nh, 0x1.cf79abc9e3b3ap-48, rh0);  // r / 2
  // p = e^r - 1 = r + 2 (r/2)^2 + r^3/6 + r^4/24, the tail in FP32 (r^3/6 is
  // below 5e-10)
  const float rf = 2.0f * d2f(rh);
  const float tail = rf * rf * rf * fma32(rf, fma32(rf, 1.0f / 120.0f, 1.0f / 24.0f), 1.0f / 6.0f);
  const double rr = rh + rh;
  const double p = fma(rr, rh, rr) + f2d(tail);
#if defined(__CUDA_ARCH__)
  const double2 tu = __ldg(reinterpret_cast<const double2 *>(kExp64) + (an.n & 255));
  double T = tu.x, U = tu.y;
#else
  double T = kExp64[an.n & 255].t, U = kExp64[an.n & 255].u;
#endif
  if (an.n >= 256) {
    const uint64_t tb = bits_of(T);
    T = double_of(static_cast<uint32_t>(tb >> 32) - (static_cast<uint32_t>(an.n >> 8) << 20),
                  static_cast<uint32_t>(tb));
    U = 1.0 - T;
  }
  const double m = fma(-T, p, U);
  const double q = fma(T, p, T);
  const double q1 = 1.0 + q;
  const double z0 = f2d_normal(an.z.h) + f2d_normal(an.z.l);
  const double z = fma(z0, fma(-q1, z0, 1.0), z0);
  const double D = k * m * q1;
  const double r0 = f2d_normal(an.rho.h) + f2d_normal(an.rho.l);
  const double dr = D * r0;
  const double er = fma(-half_of(dr), r0, 0.5);
  const double rho = fma(r0, er, r0);
  const double B = fma(4.0 * a, q * z, m);
  return kHalfSqrtG * rho * B * rk;
}

}  // namespace mr
