// Host check of csrc/dispersion.cuh against long double: prints the largest
// relative error of k and the largest error of the cosine and sine, each as a
// multiple of its bound (test_split_cpu.py).
#include <math.h>
#include <stdio.h>

#include "../mantaray_gb300/csrc/dispersion.cuh"

using namespace mr;
typedef long double Q;

static uint64_t state = 0x2545F4914F6CDD1Dull;
static double uniform() {
  state = state * 6364136223846793005ull + 1442695040888963407ull;
  return static_cast<double>(state >> 11) * 0x1p-53;
}

int main() {
  double worst_k = 0, worst_t = 0;
  int checked = 0;
  for (int i = 0; i < 300000; ++i) {
    const double period = exp(uniform() * log(1000.0) - 3.0);
    const float h = expf(static_cast<float>(uniform() * log(1e7) - 6.0));
    if (dispersion_covers(period, h)) {
      const Q w = 6.283185307179586L / static_cast<Q>(period), g = 9.8;
      const Q got = dispersion_fast(period, h);
      Q k = got;
      for (int it = 0; it < 3; ++it) {
        const Q th = tanhl(k * h);
        k -= (g * k * th - w * w) / (g * th + g * k * h * (1 - th * th));
      }
      // w, w^2 and the residual's three products: 12 units of 2^-53
      worst_k = fmax(worst_k, static_cast<double>(fabsl(got / k - 1)) / (12 * 0x1p-53));
      ++checked;
    }
    const double t = (uniform() - 0.5) * (i % 2 ? 13.0 : 2048.0);
    double c, s;
    cos_sin(t, &c, &s);
    // the table's and two sums' rounding: 4 units of 2^-53
    worst_t = fmax(worst_t, static_cast<double>(fmaxl(fabsl(c - cosl(t)), fabsl(s - sinl(t)))) /
                                (4 * 0x1p-53));
  }
  printf("%d %.4f %.4f\n", checked, worst_k, worst_t);
  return 0;
}
