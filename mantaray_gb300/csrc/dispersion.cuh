// dispersion.cuh -- |k| from the dispersion relation and the sine and cosine
// of a direction, for the device seeding (seed.cu): FP64 results from FP32 and
// float-pair (split.cuh) first approximations, 20 and 13 FP64 operations.
// Host and device code, as split.cuh.
#pragma once

#include "split.cuh"
#include "trig_table.h"

namespace mr {

constexpr double kSeedG = 9.8;  // src/wave_ray_path.rs:23

MR_HD float exp2_guess(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return exp2f(x);
#endif
}

// Whether dispersion_fast covers a period and depth (NaN: no).  The last
// condition is (kh)^2 above about 1/32: below it exp(-2kh) of the table is
// near 1 and 1 - exp(-2kh) loses relative accuracy.
MR_HD bool dispersion_covers(double period, float h) {
  return period > 0x1p-10 && period < 0x1p10 && h > 0x1p-10f && h < 0x1p20f &&
         h > 0.0078f * (d2f(period) * d2f(period));
}

// k > 0 with w2 = (2 pi / period)^2 = g k tanh(k h).  Four Newton steps in
// FP32 on a tanh a = c = w2 h / g from max(c, sqrt c) leave a relative error
// below 1e-6, one in pairs squares it, one with the residual in FP64 leaves
// FP64 rounding.  Where c > 22, tanh(kh) is 1 in FP64 and k = w2 / g.
MR_SPLIT double dispersion_fast(double period, float h) {
  // 1/period from a guess, e its residual: error e^3 ~ 2^-66
  const double r0 = f2d_normal(rcp_guess(d2f(period)));
  const double e = fma(-period, r0, 1.0);
  const double w = 6.283185307179586 * fma(r0, fma(e, e, e), r0);
  const double w2 = w * w;
  const double deep = w2 * (1.0 / kSeedG);
  const float c = d2f(deep) * h;
  if (c > 22.0f) return deep;
  float a = fmaxf(c, sqrtf(c));
  for (int it = 0; it < 4; ++it) {
    // q = exp(-2a), m = 1 - q: by the Taylor series where 1 - q would cancel
    const float x = -2.0f * a;
    float q, m;
    if (x < -0.5f) {
      q = exp2_guess(x * 1.44269504088896341f);
      m = 1.0f - q;
    } else {
      float p = fma32(x, 1.0f / 5040.0f, 1.0f / 720.0f);
      p = fma32(x, p, 1.0f / 120.0f);
      p = fma32(x, p, 1.0f / 24.0f);
      p = fma32(x, p, 1.0f / 6.0f);
      p = fma32(x, p, 0.5f);
      p = fma32(x, p, 1.0f);
      m = -(x * p);
      q = 1.0f - m;
    }
    const float z = rcp_guess(1.0f + q), th = m * z;
    a -= (a * th - c) * rcp_guess(th + a * (4.0f * q) * (z * z));
  }
  F2 k = F2{a * rcp_guess(h), 0.0f};
  // f = g k tanh(kh) - w2 in pairs; df/dk
  F2 ap = mul_f(k, h);
  int n;
  F2 q, m;
  split_exp(scale(-2.0f, ap), &n, &q, &m);
  const F2 one = fast_two_sum(1.0f, q.h);
  const F2 z = rcp2(F2{one.h, one.l + q.l});
  const F2 th = mul(m, z);
  const F2 f = add(mul(mul(F2{0x1.39999ap+3f, -0x1.99999ap-23f}, k), th), neg(to_pair(w2)));
  const float inv_df = rcp_guess(9.8f * (th.h + ap.h * (4.0f * q.h) * (z.h * z.h)));
  k = add_f(k, -((f.h + f.l) * inv_df));
  // the same residual in FP64
  const double kd = to_double(k);
  double qd, md;
  anchor_exp(kd * f2d_normal(h), n, &qd, &md);
  const double q1 = 1.0 + qd;
  const double z0 = f2d_normal(z.h) + f2d_normal(z.l);
  const double ez = fma(-q1, z0, 1.0);  // z0 is that of the k before: 1e-6 off
  const double zd = fma(z0, fma(ez, ez, ez), z0);
  const double fd = fma(kSeedG * kd, md * zd, -w2);
  return kd - f2d(d2f(fd) * inv_df);
}

// cos and sin of |t| <= 1024: t = n 2 pi/256 + r, |r| <= pi/256, cos r - 1
// and sin r by their Taylor series (the tails, below 2^-30 and r 2^-32, in
// FP32), and the angle sum with the table's values.
MR_SPLIT void cos_sin(double t, double *cos_t, double *sin_t) {
  const float nf = rintf(d2f(t) * 0x1.45f306p+5f);
  const double nd = f2d_zero(nf);
  const double r = fma(-nd, 0x1.0b4611a626331p-40, fma(-nd, 0x1.921fb544p-6, t));
  const double r2 = r * r;
  const float r2f = d2f(r2);
  const double s3 = f2d(r2f * fma32(r2f, -1.0f / 5040.0f, 1.0f / 120.0f)) - 1.0 / 6.0;
  const double s = fma(r * r2, s3, r);
  const double c = fma(r2, -0.5, f2d(r2f * r2f * fma32(r2f, -1.0f / 720.0f, 1.0f / 24.0f)));
  const int n = static_cast<int>(nf) & 255;
#if defined(__CUDA_ARCH__)
  const double2 cs = __ldg(reinterpret_cast<const double2 *>(kCosSin) + n);
  const double C = cs.x, S = cs.y;
#else
  const double C = kCosSin[n].c, S = kCosSin[n].s;
#endif
  *cos_t = C + fma(C, c, -(S * s));
  *sin_t = S + fma(S, c, C * s);
}

}  // namespace mr
