// Host check of csrc/split.cuh against long double (64 or 113 bits of
// mantissa): prints the largest error of the FP64 anchor and of the pairs'
// derivatives, each as a multiple of its bound (test_split_cpu.py).
#include <math.h>
#include <stdio.h>

#include "../mantaray_gb300/csrc/split.cuh"

using namespace mr;
typedef long double Q;

static uint64_t state = 0x9E3779B97F4A7C15ull;
static double uniform() {
  state = state * 6364136223846793005ull + 1442695040888963407ull;
  return static_cast<double>(state >> 11) * 0x1p-53;
}

int main() {
  double worst_anchor = 0, worst_pair = 0, worst_f = 0;
  int checked = 0;
  for (int i = 0; i < 300000; ++i) {
    // depths 0.01 m to 8 km, |k| 1e-3 to 3 rad/m (kh from 1e-5 to 2e4)
    Sample s = {};
    s.h = expf(static_cast<float>(log(0.01) + uniform() * log(8000 / 0.01)));
    s.g.x = 0.125f;
    const double k = exp(log(0.001) + uniform() * log(3000.0)), th = 6.283185307179586 * uniform();
    const double kx = k * cos(th), ky = k * sin(th);
    const F2 px = to_pair(kx), py = to_pair(ky);
    const V2 kv = {{px.h, py.h}, {px.l, py.l}};
    const Wave wave = wave_of(kv);
    if (!split_ok(s, wave.k2.h)) continue;
    V2 d, dk;
    double w;
    split_rhs<true>(s, wave, &d, &dk, kx, ky, &w);
    const Q g = 9.8, kk = sqrtl(static_cast<Q>(kx) * kx + static_cast<Q>(ky) * ky);
    const Q a = kk * s.h, q = expl(-2 * a), m = -expm1l(-2 * a);
    const Q rho = 1 / sqrtl(kk * m * (1 + q));
    const Q ref = sqrtl(g) / 2 * rho * (m + 4 * a * q / (1 + q)) / kk;
    const Q f = -2 * sqrtl(g) * kk * kk * q / (1 + q) * rho;
    // FP64: 16 units of 2^-53
    worst_anchor = fmax(worst_anchor, static_cast<double>(fabsl(w / ref - 1)) / 0x1p-49);
    // pairs: some 20 operations of up to 2^-46 each
    const bool xb = fabs(kx) > fabs(ky);
    const F2 dp = xb ? x_of(d) : y_of(d), df = x_of(dk);
    const Q dv = static_cast<Q>(dp.h) + dp.l;
    worst_pair = fmax(worst_pair, static_cast<double>(fabsl(dv / (ref * (xb ? kx : ky)) - 1)) / 0x1p-42);
    // f carries exp(-2a), whose relative error grows with a
    if (a < 22) {
      const Q fv = (static_cast<Q>(df.h) + df.l) / 0.125L;
      worst_f = fmax(worst_f, static_cast<double>(fabsl(fv / f - 1) / (1 + a)) / 0x1p-42);
    } else if (df.h != 0.0f) {
      worst_f = 2;
    }
    ++checked;
  }
  printf("%d %.4f %.4f %.4f\n", checked, worst_anchor, worst_pair, worst_f);
  return 0;
}
