// Device check of csrc/split.cuh's packed pairs (test_gpu_pairs.py): sums and
// differences of products on random pairs.  Prints the largest error of each,
// over |a b| + |c|, in units of 2^-43.
#include <math.h>
#include <stdio.h>

#include <vector>

#include "../mantaray_gb300/csrc/split.cuh"

using namespace mr;
constexpr int kForms = 8;

__global__ void forms(const V2 *a, const V2 *b, const V2 *c, V2 *o, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  V2 *r = o + kForms * i;
  r[0] = add(mul(a[i], b[i]), c[i]);
  r[1] = add(c[i], mul(a[i], b[i]));
  r[2] = sub(mul(a[i], b[i]), c[i]);
  r[3] = sub(c[i], mul(a[i], b[i]));
  r[4] = add(mul_f(a[i], b[i].h), c[i]);
  r[5] = sub(c[i], mul_f(a[i], b[i].h));
  r[6] = add_f(mul(a[i], b[i]), c[i].h);
  const F2 k = norm2(a[i]);
  r[7] = V2{V{k.h, k.h}, V{k.l, k.l}};
}

int main() {
  const int n = 1 << 18;
  std::vector<V2> in[3], out(kForms * n);
  V2 *dev[4];
  uint64_t state = 1;
  auto uniform = [&] {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return static_cast<double>(state >> 11) * 0x1p-52 - 1.0;
  };
  for (auto &v : in) {
    v.resize(n);
    for (V2 &q : v) {
      const F2 x = to_pair(uniform()), y = to_pair(uniform());
      q = V2{V{x.h, y.h}, V{x.l, y.l}};
    }
  }
  for (int q = 0; q < 4; ++q)
    if (cudaMalloc(&dev[q], sizeof(V2) * n * (q < 3 ? 1 : kForms)) != cudaSuccess) return 1;
  for (int q = 0; q < 3; ++q)
    cudaMemcpy(dev[q], in[q].data(), sizeof(V2) * n, cudaMemcpyHostToDevice);
  forms<<<n / 256, 256>>>(dev[0], dev[1], dev[2], dev[3], n);
  if (cudaMemcpy(out.data(), dev[3], sizeof(V2) * n * kForms, cudaMemcpyDeviceToHost) !=
      cudaSuccess)
    return 1;
  double worst[kForms] = {};
  for (int i = 0; i < n; ++i)
    for (int lane = 0; lane < 2; ++lane) {
      auto h = [&](const V2 &v) { return static_cast<double>(lane ? v.h.y : v.h.x); };
      auto all = [&](const V2 &v) { return h(v) + (lane ? v.l.y : v.l.x); };
      const double p = all(in[0][i]) * all(in[1][i]), q = all(in[0][i]) * h(in[1][i]),
                   c = all(in[2][i]), ch = h(in[2][i]);
      const F2 x = x_of(in[0][i]), y = y_of(in[0][i]);
      const double nx = static_cast<double>(x.h) + x.l, ny = static_cast<double>(y.h) + y.l;
      const double ref[kForms] = {p + c, c + p, p - c, c - p, q + c, c - q, p + ch,
                                  nx * nx + ny * ny};
      const double size[kForms] = {fabs(p) + fabs(c), fabs(p) + fabs(c), fabs(p) + fabs(c),
                                   fabs(p) + fabs(c), fabs(q) + fabs(c), fabs(q) + fabs(c),
                                   fabs(p) + fabs(ch), ref[7]};
      for (int t = 0; t < kForms; ++t)
        worst[t] = fmax(worst[t], fabs(all(out[kForms * i + t]) - ref[t]) / size[t] * 0x1p43);
    }
  for (double w : worst) printf("%.4f ", w);
  printf("\n");
  return 0;
}
