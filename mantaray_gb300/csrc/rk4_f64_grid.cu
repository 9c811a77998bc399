// rk4_f64_grid.cu -- K1 on gridded bathymetry: the plain FP64 integrator with
// the identity arithmetic, its stages on pairs of floats around one FP64
// anchor a step (split.cuh) and its lookups from per-cell records
// (split_lookup.cuh).  One ray per thread, the rows of rk4_f64.cu.
//
// A step in the domain of split_ok runs 23 (deep water) to 45 FP64
// operations instead of 190 to 370, and 1,570 to 2,200 instructions instead
// of 4,060 to 5,080.  A step that leaves that domain at any stage (a ray past
// the grid, dry or NaN nodes, k = 0) is taken again with the FP64 form of
// ray_exact.cuh, which also decides how the ray stops: NaN rows and row
// counts are that form's.  Every ray's arithmetic depends on its own state
// only, so a ray's rows are the same in every call.
//
// Bounds: few rays, the dependent chain of a step (FP32 4.3 cycles a link,
// FP64 64); many rays, the chain and the issue slots (55% busy, the FP64 pipe
// 51%, at the 13.5 warps an SM that 65,536 rays give).  128 registers: 7
// blocks of 64 per SM are what 65,536 rays need to be resident at once; with
// 156 they ran in two waves, 24 ms against 15 for the same code.
//
// Measured against the FP64 form (GB300, full trajectories): the seamount,
// 65,536 rays x 2,000 steps, 59.7 -> 12.4 ms (2.19 -> 10.5 G ray-steps/s);
// the planar beach, 1,024 rays x 2,000 steps, 41.3 -> 9.4 ms; one ray x 200
// steps 3.77 -> 0.84 ms.  Against the model in 64 bits the trajectories'
// error is unchanged (seamount 5e-12, beach 4e-10: the lookups' f32
// interpolation).  Against the same lookups with the rest in 80-bit
// arithmetic (800 rays x 500 to 1,000 steps over a shoal and a jet) the
// positions' median error is 1.03-1.04 times the FP64 form's, 3.2e-11 and
// 4.6e-11 m, of which the rounding of the FP64 state is nearly all.

#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "ray_exact.cuh"
#include "split_lookup.cuh"

namespace mr {

namespace {

struct StepConst {
  double dt, half, sixth;
  F2 dt2, half2, sixth2;  // the same as pairs
};

// The FP64 form's step from y (ray_exact.cuh, rk4_f64.cu).  Returns whether
// the ray stops after it.
__device__ __noinline__ bool fp64_step(const BathyDev &b, const CurrentDev &c, double dt,
                                       double *yio) {
  double y[4], k1[4], kc[4], acc[4], in[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) y[q] = yio[q];
  system<RhsIdentity, NoCache>(b, c, y, k1);
#pragma unroll
  for (int q = 0; q < 4; ++q) acc[q] = kc[q] = k1[q];
#pragma unroll 1
  for (int st = 0; st < 3; ++st) {
    const double hs = st == 2 ? dt : dt / 2.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) in[q] = fma(kc[q], hs, y[q]);
    system<RhsIdentity, NoCache>(b, c, in, kc);
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = st < 2 ? fma(kc[q], 2.0, acc[q]) : acc[q] + kc[q];
  }
  const double sixth = dt / 6.0;
#pragma unroll
  for (int q = 0; q < 4; ++q) y[q] = fma(acc[q], sixth, y[q]);
#pragma unroll
  for (int q = 0; q < 4; ++q) yio[q] = y[q];
  return all_nan4(k1) || all_nan4(y);
}

// Whether the derivative at y is all NaN (MR_STOP_FRESH's test).
__device__ __noinline__ bool fp64_stopped(const BathyDev &b, const CurrentDev &c,
                                          const double *y) {
  double s[4], k[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) s[q] = y[q];
  system<RhsIdentity, NoCache>(b, c, s, k);
  return all_nan4(k);
}

// f32 coordinates of the position (h + m + r) + inc: RN of the sum, as the
// FP64 form rounds its stage positions.  The remainder R carries 24 bits; a
// sum whose rounding they do not decide (1 in 10^6) returns false.
__device__ __forceinline__ bool stage_point(const V &h, const V &m, const V &r, const V2 &inc,
                                            V *out) {
  const V2 s = two_sum(inc.h, m);
  const V2 t = two_sum(h, s.h);
  const V R = vadd(t.l, vadd(s.l, vadd(inc.l, r)));
  const V a = vfma(R, both(1.0f + 0x1p-20f), t.h), b = vfma(R, both(1.0f - 0x1p-20f), t.h);
  *out = a;
  return a.x == b.x && a.y == b.y;
}

// One step in pairs; false (y unchanged) when any stage is outside split_ok.
// The last three stages run in a rolled loop: two copies of the lookups and
// of the right-hand side, which the instruction cache holds (the loop
// unrolled is 1.6x slower).
template <int CUR>
__device__ __forceinline__ bool split_step(const BathyDev &b, const CurrentDev &c,
                                           const StepConst &h, SplitCell<CUR> &C, double y[4]) {
  V xh, xm, xr;
  split3(y[0], &xh.x, &xm.x, &xr.x);
  split3(y[1], &xh.y, &xm.y, &xr.y);
  const F2 kx = to_pair(y[2]), ky = to_pair(y[3]);
  const V2 k = V2{V{kx.h, ky.h}, V{kx.l, ky.l}};
  Wave wv = wave_of(k);
  Sample s;
  if (!split_sample<CUR>(b, c, d2f(y[0]), d2f(y[1]), [&](double *px, double *py) {
        *px = y[0];
        *py = y[1];
      }, C, s))
    return false;
  bool ok = split_ok(s, wv.k2.h);
  V2 d1, d, dk;
  double w;
  split_rhs<true>(s, wv, &d1, &dk, y[2], y[3], &w);
  // gridded currents are f32 values: their low halves are 0
  const double ax = fma(w, y[2], CUR == SPLIT_CONSTANT ? c.cu : f2d(s.uv.h.x));
  const double ay = fma(w, y[3], CUR == SPLIT_CONSTANT ? c.cv : f2d(s.uv.h.y));
  V2 sd = zero2(), sk = dk;               // weighted sums of d - d1 and of dk
  d = d1;
#pragma unroll 1
  for (int st = 0; st < 3; ++st) {
    if (!ok) return false;  // tested where the branches already are
    const F2 hs = st == 2 ? h.dt2 : h.half2;
    wv = wave_of(add(k, mul(dk, both(hs))));
    V t;
    auto at = [&](double *px, double *py) {
      const double hd = st == 2 ? h.dt : h.half;
      *px = fma(hd, to_double(x_of(d)), y[0]);
      *py = fma(hd, to_double(y_of(d)), y[1]);
    };
    if (!stage_point(xh, xm, xr, mul(d, both(hs)), &t)) {
      double px, py;
      at(&px, &py);
      t = V{d2f(px), d2f(py)};
    }
    if (!split_sample<CUR>(b, c, t.x, t.y, at, C, s)) return false;
    ok = split_ok(s, wv.k2.h);
    split_rhs<false>(s, wv, &d, &dk, 0.0, 0.0, nullptr);
    const float wt = st == 2 ? 1.0f : 2.0f;
    sd = add(sd, scale(wt, sub(d, d1)));
    sk = add(sk, scale(wt, dk));
  }
  if (!ok) return false;
  const V2 e = mul(sd, both(h.sixth2));
  y[0] += fma(h.dt, ax, f2d_zero(e.h.x)) + f2d_zero(e.l.x);
  y[1] += fma(h.dt, ay, f2d_zero(e.h.y)) + f2d_zero(e.l.y);
  y[2] = fma(h.sixth, to_double(x_of(sk)), y[2]);
  y[3] = fma(h.sixth, to_double(y_of(sk)), y[3]);
  return true;
}

template <int STOP_RULE, int CUR>
__global__ void __launch_bounds__(kK1Block, 8)
    rk4_f64_grid_kernel(const __grid_constant__ BathyDev b, const __grid_constant__ CurrentDev c,
                        const __grid_constant__ TraceArgs a, const StepConst h) {
  const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const bool valid = i < a.n;
  const unsigned warp_mask = blockDim.x >= 32 ? 0xffffffffu : (1u << blockDim.x) - 1u;
  SplitCell<CUR> C;
  split_start<CUR>(c, C);
  const uint64_t plane = a.rows_cap * a.n;
  double y[4] = {0.0, 0.0, 0.0, 0.0};
  double t = a.t0;
  bool alive = valid;
  uint64_t rows = 0;
  if (valid) {
    y[0] = a.x0[i]; y[1] = a.y0[i]; y[2] = a.kx0[i]; y[3] = a.ky0[i];
    store_row(a.traj, plane, a.n, 0, i, t, y);
    rows = 1;
  }
  uint64_t s = 0;
  for (; s < a.nsteps; ++s) {
    // Once every lane of the warp has stopped, the rest is NaN padding.
    if (__all_sync(warp_mask, !alive)) break;
    bool stop = false;
    if (alive && !split_step<CUR>(b, c, h, C, y)) {
      double v[4] = {y[0], y[1], y[2], y[3]};
      if (STOP_RULE == 1 && s > 0 && fp64_stopped(b, c, v)) {
        alive = false;  // the previous step's new state has no derivative
      } else {
        stop = fp64_step(b, c, h.dt, v);
#pragma unroll
        for (int q = 0; q < 4; ++q) y[q] = v[q];
      }
    }
    if (alive) {
      t = t + h.dt;
      store_row(a.traj, plane, a.n, s + 1, i, t, y);
      ++rows;
      if (stop) alive = false;
    } else if (valid) {
      store_nan_row(a.traj, plane, a.n, s + 1, i);
    }
  }
  if (STOP_RULE == 1 && alive && a.nsteps > 0) {
    double v[4] = {y[0], y[1], y[2], y[3]};
    if (fp64_stopped(b, c, v)) alive = false;
  }
  if (valid) {
    for (uint64_t row = rows > s + 1 ? rows : s + 1; row < a.rows_cap; ++row)
      store_nan_row(a.traj, plane, a.n, row, i);
    a.n_rows[i] = static_cast<int32_t>(rows);
    a.status[i] = alive ? 0 : 1;
  }
}

// ----------------------------------------------------------- the records --

__device__ __forceinline__ bool small_gradient(double g) {
  return g > -1048576.0 && g < 1048576.0;  // false for NaN
}

// One record per cell (fields.h): what cell_prepare (lookup.cuh) computes,
// with the same operations.  A cell whose gradients are outside the pairs'
// domain gets a NaN coefficient, which sends its rays to the FP64 form.
__global__ void build_bathy_records(BathyDev b, float4 *rec) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t nx = static_cast<int64_t>(b.nx), ny = static_cast<int64_t>(b.ny);
  if (k >= nx * ny) return;
  const int64_t i = k % nx, j = k / nx;
  if (i + 1 >= nx || j + 1 >= ny) return;
  const float sw = b.depth32[k], nw = b.depth32[k + nx], ne = b.depth32[k + nx + 1],
              se = b.depth32[k + 1];
  CellWeights<1> W;
  const float pv[1][4] = {{sw, nw, ne, se}};
  float4 r0, r1;
  if (cell_prepare<1>(b.x[i], b.x[i + 1], b.y[j], b.y[j + 1], pv, W) &&
      small_gradient(b.gx[k]) && small_gradient(b.gy[k])) {
    r0 = make_float4(W.a00[0], W.a10[0], W.a01[0], W.a11[0]);
    r1 = make_float4(b.gx[k], b.gy[k], W.m01, W.m10);
  } else {
    r0 = r1 = make_float4(f32_nan(), 0.0f, 0.0f, 0.0f);
  }
  rec[2 * k] = r0;
  rec[2 * k + 1] = r1;
}

__global__ void build_current_records(CurrentDev c, float4 *rec) {
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t nx = static_cast<int64_t>(c.nx), ny = static_cast<int64_t>(c.ny);
  if (k >= nx * ny) return;
  const int64_t i = k % nx, j = k / nx;
  if (i + 1 >= nx || j + 1 >= ny) return;
  const float pv[2][4] = {{c.u32[k], c.u32[k + nx], c.u32[k + nx + 1], c.u32[k + 1]},
                          {c.v32[k], c.v32[k + nx], c.v32[k + nx + 1], c.v32[k + 1]}};
  const double g[4] = {c.dudx[k], c.dudy[k], c.dvdx[k], c.dvdy[k]};
  CellWeights<2> W;
  const bool ok = cell_prepare<2>(c.x32[i], c.x32[i + 1], c.y32[j], c.y32[j + 1], pv, W) &&
                  small_gradient(g[0]) && small_gradient(g[1]) && small_gradient(g[2]) &&
                  small_gradient(g[3]);
  float4 *r = rec + 5 * k;
  if (!ok) {
    r[0] = r[1] = make_float4(f32_nan(), f32_nan(), 0.0f, 0.0f);
    r[2] = r[3] = r[4] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    return;
  }
  r[0] = make_float4(W.a00[0], W.a00[1], W.a10[0], W.a10[1]);
  r[1] = make_float4(W.a01[0], W.a01[1], W.a11[0], W.a11[1]);
  const F2 ux = to_pair(g[0]), uy = to_pair(g[1]), vx = to_pair(g[2]), vy = to_pair(g[3]);
  r[2] = make_float4(ux.h, uy.h, ux.l, uy.l);
  r[3] = make_float4(vx.h, vy.h, vx.l, vy.l);
  r[4] = make_float4(W.m01, W.m10, 0.0f, 0.0f);
}

F2 host_pair(double v) {
  const float h = static_cast<float>(v);
  return F2{h, static_cast<float>(v - static_cast<double>(h))};
}

template <int STOP_RULE>
void launch_cur(int cur, unsigned grid, int block, const BathyDev &b, const CurrentDev &c,
                const TraceArgs &a, const StepConst &h, cudaStream_t s) {
  if (cur == SPLIT_CONSTANT)
    rk4_f64_grid_kernel<STOP_RULE, SPLIT_CONSTANT><<<grid, block, 0, s>>>(b, c, a, h);
  else if (cur == SPLIT_GRID)
    rk4_f64_grid_kernel<STOP_RULE, SPLIT_GRID><<<grid, block, 0, s>>>(b, c, a, h);
  else
    rk4_f64_grid_kernel<STOP_RULE, SPLIT_SAME><<<grid, block, 0, s>>>(b, c, a, h);
}

}  // namespace

cudaError_t launch_bathy_records(const BathyDev &b, void *rec, cudaStream_t stream) {
  const uint64_t cells = b.nx * b.ny;
  build_bathy_records<<<static_cast<unsigned>((cells + 255) / 256), 256, 0, stream>>>(
      b, static_cast<float4 *>(rec));
  return cudaGetLastError();
}

cudaError_t launch_current_records(const CurrentDev &c, void *rec, cudaStream_t stream) {
  const uint64_t cells = c.nx * c.ny;
  build_current_records<<<static_cast<unsigned>((cells + 255) / 256), 256, 0, stream>>>(
      c, static_cast<float4 *>(rec));
  return cudaGetLastError();
}

// The pairs' exponent range bounds the step too.
bool split_covers(const BathyDev &b, const CurrentDev &c, const TraceArgs &a) {
  const double dt = a.dt < 0.0 ? -a.dt : a.dt;
  const bool current = c.kind == CURRENT_GRID ? c.split.rec != nullptr
                                              : c.cu == c.cu && c.cv == c.cv;
  return b.kind == BATHY_GRID && b.split.rec && current && dt > 0x1p-40 && dt < 0x1p40;
}

cudaError_t launch_rk4_f64_grid(const BathyDev &b, const CurrentDev &c, const TraceArgs &a,
                                int stop_rule, int same_axes, unsigned grid, int block,
                                cudaStream_t stream) {
  StepConst h;
  h.dt = a.dt;
  h.half = a.dt / 2.0;
  h.sixth = a.dt / 6.0;
  h.dt2 = host_pair(h.dt);
  h.half2 = host_pair(h.half);
  h.sixth2 = host_pair(h.sixth);
  const int cur = c.kind != CURRENT_GRID ? SPLIT_CONSTANT : same_axes ? SPLIT_SAME : SPLIT_GRID;
  if (stop_rule == 1)
    launch_cur<1>(cur, grid, block, b, c, a, h, stream);
  else
    launch_cur<0>(cur, grid, block, b, c, a, h, stream);
  return cudaGetLastError();
}

}  // namespace mr
