// diff.cu -- K3 (discrete adjoint) and K4 (tangent-linear) of the RK4 ray
// integrator, with its forward pass (checkpoints every C steps).
//
// The differentiated map is the reference's RK4 step (ode_solvers 0.4.0, as
// restated for the plain form) over the reference's equations
// (src/wave_ray_path.rs:118-216) with the grid lookups in the working
// precision T, without the reference's f32 casts (those make the map a
// staircase at the ulp level, below any finite-difference step): bilinear
// depth / current inside the cell that holds the point (the reference's
// corner rule), and cell-constant forward-difference gradients
// (src/bathymetry/cartesian_netcdf3.rs:119-134,
// src/current/cartesian_current.rs:515-536).  Inside a cell the map is smooth;
// cell-constant gradients jump across cell edges, where it is not
// differentiable.
//
// Right-hand side F(s; D, U, V) with s = (x, y, kx, ky), k = |(kx, ky)|,
// c = kx/k, s_ = ky/k, a = k h, and the group velocity q(k, h) and refraction
// factor f(k, h) = -k sigma / sinh(2a), sigma = sqrt(g k tanh a):
//   F0 = q c + u,  F1 = q s_ + v,
//   F2 = f hx - kx ux - ky vx,  F3 = f hy - kx uy - ky vy.
// Its partial derivatives are written out by hand below (q_k, q_h, f_k, f_h
// from sigma and n(a) = 1 + 2a / sinh(2a), with exp(-2a) forms that stay finite
// in deep water); the tangent-linear step applies them forward (JVP), the
// adjoint step backward (VJP), both through the four RK4 stages.
//
// Adjoint pass per ray: the forward stored the state every C steps; each
// segment is recomputed from its checkpoint into a scratch buffer (every
// step's four stage states) and walked backward, evaluating each stage's
// partials where its transpose is applied.  Gradients with respect to grid
// nodes are accumulated per ray while the ray stays in one cell, then added to
// the node arrays with FP64 atomics, aggregated across the lanes of a warp that
// flush the same cell.  The per-cell accumulation runs in the working
// precision; only the accumulation onto the node arrays is FP64.
//
// The recomputed states need not be the forward's to the last bit (the forward
// may have run on pairs and this pass not, or the other way round), so a stage
// beside a grid's edge can have no derivative here.  The ray's walk backward
// ends there: no cell of that stage is read or added to, and the gradient
// returned is that of the state it had come to.
//
// In FP64 all three run on float pairs where diff_split.cu covers the call; the
// kernels here in double serve the rest (few steps, where the records cost more
// than they save, a stream under capture, grids beyond its limits).

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/mantaray_gpu.h"
#include "diff.cuh"
#include "diff_split.h"
#include "handles.h"

namespace mr {
namespace {

// ------------------------------------------------------------- kernels --

template <typename T>
__global__ void __launch_bounds__(64) diff_forward_kernel(DiffArgs<T> A) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  T y[4] = {A.x0[i], A.y0[i], A.kx0[i], A.ky0[i]};
  bool ok = true;
  Held<T> N;
  for (int64_t s = 0; s < A.steps; ++s) {
    if (s % A.ck_every == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) A.ckpt[((s / A.ck_every) * 4 + q) * A.n + i] = y[q];
    }
    if (!rk4(A, y, N)) {
      ok = false;
      break;
    }
  }
  const T nan = T(NAN);
#pragma unroll
  for (int q = 0; q < 4; ++q) A.end_state[q * A.n + i] = ok ? y[q] : nan;
  A.status[i] = ok ? 0 : 1;
}

template <typename T>
__global__ void __launch_bounds__(64) diff_tangent_kernel(DiffArgs<T> A) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  T y[4] = {A.x0[i], A.y0[i], A.kx0[i], A.ky0[i]};
  T dy[4] = {A.dstate0[i], A.dstate0[A.n + i], A.dstate0[2 * A.n + i], A.dstate0[3 * A.n + i]};
  bool ok = true;
  Held<T> N;
  const T half = A.dt * T(0.5), sixth = A.dt / T(6);
  for (int64_t s = 0; s < A.steps && ok; ++s) {
    Point<T> P;
    T k1[4], k2[4], k3[4], k4[4], d1[4], d2[4], d3[4], d4[4], t[4], dt_[4];
    ok = eval(A, y, P, k1, N);
    if (ok) jvp(A, y, P, dy, d1);
#pragma unroll
    for (int q = 0; q < 4; ++q) { t[q] = y[q] + k1[q] * half; dt_[q] = dy[q] + d1[q] * half; }
    ok = ok && eval(A, t, P, k2, N);
    if (ok) jvp(A, t, P, dt_, d2);
#pragma unroll
    for (int q = 0; q < 4; ++q) { t[q] = y[q] + k2[q] * half; dt_[q] = dy[q] + d2[q] * half; }
    ok = ok && eval(A, t, P, k3, N);
    if (ok) jvp(A, t, P, dt_, d3);
#pragma unroll
    for (int q = 0; q < 4; ++q) { t[q] = y[q] + k3[q] * A.dt; dt_[q] = dy[q] + d3[q] * A.dt; }
    ok = ok && eval(A, t, P, k4, N);
    if (ok) {
      jvp(A, t, P, dt_, d4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        y[q] = y[q] + (((k1[q] + k2[q] * T(2)) + k3[q] * T(2)) + k4[q]) * sixth;
        dy[q] = dy[q] + (((d1[q] + d2[q] * T(2)) + d3[q] * T(2)) + d4[q]) * sixth;
      }
    }
  }
  const T nan = T(NAN);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    A.end_state[q * A.n + i] = ok ? y[q] : nan;
    A.d_end[q * A.n + i] = ok ? dy[q] : nan;
  }
  A.status[i] = ok ? 0 : 1;
}

// The stages run in rolled loops (unrolled, instruction fetch was the bound:
// 7.8 ms against 7.0 for 131,071 rays x 300 steps in FP32), each reading the
// next one's state ahead.  FP32: 128 registers, 8 blocks of 64 per SM (7 blocks
// 7.2 ms, 9 8.7, 10 9.4: what does not fit is spilled); 3,100 instructions a
// warp-step at 59% of the issue slots bound it.  FP64 takes what it needs.
template <typename T>
__global__ void __launch_bounds__(64, sizeof(T) == 4 ? 8 : 1) diff_adjoint_kernel(DiffArgs<T> A) {
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= A.n) return;
  if (A.status[i] != 0) {  // no gradient through a ray that stopped
#pragma unroll
    for (int q = 0; q < 4; ++q) A.grad_state0[q * A.n + i] = T(0);
    return;
  }
  T lam[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) lam[q] = A.grad_end[q * A.n + i];
  NodeAcc<T> acc;
  acc.bkey = acc.ckey = -1;
#pragma unroll
  for (int q = 0; q < 4; ++q) acc.d[q] = acc.u[q] = acc.v[q] = T(0);
  Held<T> N;
  const T half = A.dt * T(0.5), h = A.dt, sixth = A.dt / T(6), third = A.dt / T(3);
  for (int64_t seg = A.n_ck - 1; seg >= 0; --seg) {
    const int64_t first = seg * A.ck_every;
    const int64_t last = min(first + A.ck_every, A.steps);  // steps [first, last)
    // recompute the segment from its checkpoint, keeping every step's four
    // stage states (y, Y2, Y3, Y4) in the scratch
    T y[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) y[q] = A.ckpt[(seg * 4 + q) * A.n + i];
    for (int64_t s = first; s < last; ++s) {
      T *row = A.seg + (s - first) * 16 * A.n + i;
      T Y[4], sum[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
      for (int q = 0; q < 4; ++q) Y[q] = y[q];
#pragma unroll 1
      for (int st = 0; st < 4; ++st) {
#pragma unroll
        for (int q = 0; q < 4; ++q) row[(4 * st + q) * A.n] = Y[q];
        if (st == 3 && s + 1 == last) break;  // the last step's end is not needed
        Point<T> P;
        T k[4];
        if (!eval(A, Y, P, k, N)) goto done;
        const T wt = st == 0 || st == 3 ? T(1) : T(2), f = st == 2 ? h : half;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          sum[q] = sum[q] + k[q] * wt;
          Y[q] = y[q] + k[q] * f;
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) y[q] = y[q] + sum[q] * sixth;
    }
    // walk it backward: each stage's partials are evaluated where its
    // transpose is applied (one live Point)
    T Yn[4];  // the next stage state, read ahead
    for (int64_t s = last - 1; s >= first; --s) {
      const T *row = A.seg + (s - first) * 16 * A.n + i;
      T r[4], r4[4], r3[4], r2[4];
#pragma unroll 1
      for (int st = 3; st >= 0; --st) {
        Point<T> P;
        T kd[4], w[4], Y[4];
        if (st == 3 && s == last - 1) {
#pragma unroll
          for (int q = 0; q < 4; ++q) Y[q] = row[(12 + q) * A.n];
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) Y[q] = Yn[q];
        }
        if (st > 0 || s > first) {
          const T *ahead = row + 4 * (st - 1) * A.n;  // of the step before for st = 0
#pragma unroll
          for (int q = 0; q < 4; ++q) Yn[q] = ahead[q * A.n];
        }
        if (!eval(A, Y, P, kd, N)) goto done;
        const T c = st == 3 || st == 0 ? sixth : third, f = st == 2 ? h : half;
        if (st == 3) {
#pragma unroll
          for (int q = 0; q < 4; ++q) w[q] = lam[q] * c;
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) w[q] = lam[q] * c + f * r[q];
        }
        vjp(A, Y, P, w, r, acc);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (st == 3) r4[q] = r[q];
          if (st == 2) r3[q] = r[q];
          if (st == 1) r2[q] = r[q];
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) lam[q] = lam[q] + r[q] + r2[q] + r3[q] + r4[q];
    }
  }
done:
  flush_bathy(A, acc);
  flush_current(A, acc);
#pragma unroll
  for (int q = 0; q < 4; ++q) A.grad_state0[q * A.n + i] = lam[q];
}

constexpr int kDiffBlock = 64;

template <typename T>
int make_args(const mr_diff_grid *bgrid, const void *depth, const mr_diff_grid *cgrid,
              const void *u, const void *v, size_t n, const void *x0, const void *y0,
              const void *kx0, const void *ky0, double dt, int64_t steps, int64_t ck_every,
              DiffArgs<T> *A) {
  if (!bgrid || !cgrid || !depth || !u || !v)
    return fail(MR_ERR_INVALID_ARGUMENT, "null grid or field");
  if (bgrid->nx < 2 || bgrid->ny < 2 || cgrid->nx < 2 || cgrid->ny < 2 ||
      bgrid->nx > INT32_MAX || bgrid->ny > INT32_MAX || cgrid->nx > INT32_MAX ||
      cgrid->ny > INT32_MAX)
    return fail(MR_ERR_INVALID_ARGUMENT, "grids need 2 to 2^31-1 points per axis");
  if (!(bgrid->dx > 0) || !(bgrid->dy > 0) || !(cgrid->dx > 0) || !(cgrid->dy > 0))
    return fail(MR_ERR_INVALID_ARGUMENT, "grid spacing must be positive");
  if (n > 0 && (!x0 || !y0 || !kx0 || !ky0)) return fail(MR_ERR_INVALID_ARGUMENT, "null rays");
  if (steps < 0 || ck_every < 1 || !(dt > 0.0))
    return fail(MR_ERR_INVALID_ARGUMENT, "steps >= 0, checkpoint_every >= 1, dt > 0 needed");
  *A = DiffArgs<T>{};
  A->bg = DGrid<T>{static_cast<const T *>(depth), nullptr, static_cast<int>(bgrid->nx),
                   static_cast<int>(bgrid->ny), T(bgrid->x0), T(bgrid->y0), T(1.0 / bgrid->dx),
                   T(1.0 / bgrid->dy)};
  A->cg = DGrid<T>{static_cast<const T *>(u), static_cast<const T *>(v), static_cast<int>(cgrid->nx),
                   static_cast<int>(cgrid->ny), T(cgrid->x0), T(cgrid->y0), T(1.0 / cgrid->dx),
                   T(1.0 / cgrid->dy)};
  A->same_grid = bgrid->nx == cgrid->nx && bgrid->ny == cgrid->ny && bgrid->x0 == cgrid->x0 &&
                 bgrid->y0 == cgrid->y0 && bgrid->dx == cgrid->dx && bgrid->dy == cgrid->dy;
  A->n = static_cast<int64_t>(n);
  A->x0 = static_cast<const T *>(x0);
  A->y0 = static_cast<const T *>(y0);
  A->kx0 = static_cast<const T *>(kx0);
  A->ky0 = static_cast<const T *>(ky0);
  A->dt = T(dt);
  A->steps = steps;
  A->ck_every = ck_every;
  A->n_ck = steps == 0 ? 0 : (steps + ck_every - 1) / ck_every;
  return MR_OK;
}

// The same call for the kernels on pairs (diff_split.cu).
DiffCall split_call(const DiffArgs<double> &A) {
  DiffCall c{};
  c.depth = A.bg.a; c.u = A.cg.a; c.v = A.cg.b;
  c.bnx = A.bg.nx; c.bny = A.bg.ny; c.cnx = A.cg.nx; c.cny = A.cg.ny;
  c.bx0 = A.bg.x0; c.by0 = A.bg.y0; c.b_inv_dx = A.bg.inv_dx; c.b_inv_dy = A.bg.inv_dy;
  c.cx0 = A.cg.x0; c.cy0 = A.cg.y0; c.c_inv_dx = A.cg.inv_dx; c.c_inv_dy = A.cg.inv_dy;
  c.same_grid = A.same_grid;
  c.n = A.n; c.steps = A.steps; c.ck_every = A.ck_every; c.n_ck = A.n_ck;
  c.x0 = A.x0; c.y0 = A.y0; c.kx0 = A.kx0; c.ky0 = A.ky0;
  c.dt = A.dt;
  c.ckpt = A.ckpt; c.end_state = A.end_state; c.status = A.status;
  c.grad_end = A.grad_end; c.seg = A.seg; c.grad_state0 = A.grad_state0;
  c.grad_depth = A.grad_depth; c.grad_u = A.grad_u; c.grad_v = A.grad_v;
  c.dstate0 = A.dstate0; c.d_depth = A.d_depth; c.d_u = A.d_u; c.d_v = A.d_v;
  c.d_end = A.d_end;
  return c;
}

unsigned blocks_for(size_t n) { return static_cast<unsigned>((n + kDiffBlock - 1) / kDiffBlock); }

}  // namespace
}  // namespace mr

using mr::cuda_fail;
using mr::fail;

extern "C" {

int mr_diff_forward(int precision, const mr_diff_grid *bgrid, const void *depth,
                    const mr_diff_grid *cgrid, const void *u, const void *v, size_t n,
                    const void *x0, const void *y0, const void *kx0, const void *ky0, double dt,
                    int64_t steps, int64_t checkpoint_every, void *checkpoints, void *end_state,
                    uint8_t *status, void *stream) {
  cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : cudaStreamPerThread;
  if (n > 0 && (!end_state || !status || (steps > 0 && !checkpoints)))
    return fail(MR_ERR_INVALID_ARGUMENT, "null output");
  if (precision == 64) {
    mr::DiffArgs<double> A;
    int rc = mr::make_args(bgrid, depth, cgrid, u, v, n, x0, y0, kx0, ky0, dt, steps,
                           checkpoint_every, &A);
    if (rc) return rc;
    if (n == 0) return MR_OK;
    A.ckpt = static_cast<double *>(checkpoints);
    A.end_state = static_cast<double *>(end_state);
    A.status = status;
    cudaError_t se = cudaSuccess;
    if (mr::launch_diff_split(mr::DIFF_FORWARD, mr::split_call(A), s, &se))
      return se == cudaSuccess ? MR_OK : cuda_fail(se, "diff_forward launch");
    mr::diff_forward_kernel<double><<<mr::blocks_for(n), mr::kDiffBlock, 0, s>>>(A);
  } else if (precision == 32) {
    mr::DiffArgs<float> A;
    int rc = mr::make_args(bgrid, depth, cgrid, u, v, n, x0, y0, kx0, ky0, dt, steps,
                           checkpoint_every, &A);
    if (rc) return rc;
    if (n == 0) return MR_OK;
    A.ckpt = static_cast<float *>(checkpoints);
    A.end_state = static_cast<float *>(end_state);
    A.status = status;
    mr::diff_forward_kernel<float><<<mr::blocks_for(n), mr::kDiffBlock, 0, s>>>(A);
  } else {
    return fail(MR_ERR_INVALID_ARGUMENT, "precision must be 64 or 32");
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MR_OK : cuda_fail(e, "diff_forward launch");
}

int mr_diff_backward(int precision, const mr_diff_grid *bgrid, const void *depth,
                     const mr_diff_grid *cgrid, const void *u, const void *v, size_t n,
                     const void *x0, const void *y0, const void *kx0, const void *ky0, double dt,
                     int64_t steps, int64_t checkpoint_every, const void *checkpoints,
                     const uint8_t *status, const void *grad_end, void *segment,
                     void *grad_state0, double *grad_depth, double *grad_u, double *grad_v,
                     void *stream) {
  cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : cudaStreamPerThread;
  if (!grad_depth || !grad_u || !grad_v) return fail(MR_ERR_INVALID_ARGUMENT, "null gradient array");
  if (n > 0 && (!status || !grad_end || !grad_state0 || (steps > 0 && (!checkpoints || !segment))))
    return fail(MR_ERR_INVALID_ARGUMENT, "null argument");
  const size_t bnodes = bgrid ? bgrid->nx * bgrid->ny : 0;
  const size_t cnodes = cgrid ? cgrid->nx * cgrid->ny : 0;
  cudaError_t e = cudaSuccess;
  if (precision == 64) {
    mr::DiffArgs<double> A;
    int rc = mr::make_args(bgrid, depth, cgrid, u, v, n, x0, y0, kx0, ky0, dt, steps,
                           checkpoint_every, &A);
    if (rc) return rc;
    A.ckpt = const_cast<double *>(static_cast<const double *>(checkpoints));
    A.status = const_cast<uint8_t *>(status);
    A.grad_end = static_cast<const double *>(grad_end);
    A.seg = static_cast<double *>(segment);
    A.grad_state0 = static_cast<double *>(grad_state0);
    A.grad_depth = grad_depth; A.grad_u = grad_u; A.grad_v = grad_v;
    e = cudaMemsetAsync(grad_depth, 0, bnodes * sizeof(double), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(grad_u, 0, cnodes * sizeof(double), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(grad_v, 0, cnodes * sizeof(double), s);
    if (e == cudaSuccess && n > 0 &&
        !mr::launch_diff_split(mr::DIFF_ADJOINT, mr::split_call(A), s, &e))
      mr::diff_adjoint_kernel<double><<<mr::blocks_for(n), mr::kDiffBlock, 0, s>>>(A);
  } else if (precision == 32) {
    mr::DiffArgs<float> A;
    int rc = mr::make_args(bgrid, depth, cgrid, u, v, n, x0, y0, kx0, ky0, dt, steps,
                           checkpoint_every, &A);
    if (rc) return rc;
    A.ckpt = const_cast<float *>(static_cast<const float *>(checkpoints));
    A.status = const_cast<uint8_t *>(status);
    A.grad_end = static_cast<const float *>(grad_end);
    A.seg = static_cast<float *>(segment);
    A.grad_state0 = static_cast<float *>(grad_state0);
    A.grad_depth = grad_depth; A.grad_u = grad_u; A.grad_v = grad_v;
    e = cudaMemsetAsync(grad_depth, 0, bnodes * sizeof(double), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(grad_u, 0, cnodes * sizeof(double), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(grad_v, 0, cnodes * sizeof(double), s);
    if (e == cudaSuccess && n > 0)
      mr::diff_adjoint_kernel<float><<<mr::blocks_for(n), mr::kDiffBlock, 0, s>>>(A);
  } else {
    return fail(MR_ERR_INVALID_ARGUMENT, "precision must be 64 or 32");
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? MR_OK : cuda_fail(e, "diff_adjoint launch");
}

int mr_diff_tangent(int precision, const mr_diff_grid *bgrid, const void *depth,
                    const mr_diff_grid *cgrid, const void *u, const void *v, size_t n,
                    const void *x0, const void *y0, const void *kx0, const void *ky0,
                    const void *dstate0, const void *d_depth, const void *d_u, const void *d_v,
                    double dt, int64_t steps, void *end_state, void *d_end, uint8_t *status,
                    void *stream) {
  cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : cudaStreamPerThread;
  if (n > 0 && (!dstate0 || !end_state || !d_end || !status))
    return fail(MR_ERR_INVALID_ARGUMENT, "null argument");
  if (precision == 64) {
    mr::DiffArgs<double> A;
    int rc = mr::make_args(bgrid, depth, cgrid, u, v, n, x0, y0, kx0, ky0, dt, steps, 1, &A);
    if (rc) return rc;
    if (n == 0) return MR_OK;
    A.dstate0 = static_cast<const double *>(dstate0);
    A.d_depth = static_cast<const double *>(d_depth);
    A.d_u = static_cast<const double *>(d_u);
    A.d_v = static_cast<const double *>(d_v);
    A.end_state = static_cast<double *>(end_state);
    A.d_end = static_cast<double *>(d_end);
    A.status = status;
    cudaError_t se = cudaSuccess;
    if (mr::launch_diff_split(mr::DIFF_TANGENT, mr::split_call(A), s, &se))
      return se == cudaSuccess ? MR_OK : cuda_fail(se, "diff_tangent launch");
    mr::diff_tangent_kernel<double><<<mr::blocks_for(n), mr::kDiffBlock, 0, s>>>(A);
  } else if (precision == 32) {
    mr::DiffArgs<float> A;
    int rc = mr::make_args(bgrid, depth, cgrid, u, v, n, x0, y0, kx0, ky0, dt, steps, 1, &A);
    if (rc) return rc;
    if (n == 0) return MR_OK;
    A.dstate0 = static_cast<const float *>(dstate0);
    A.d_depth = static_cast<const float *>(d_depth);
    A.d_u = static_cast<const float *>(d_u);
    A.d_v = static_cast<const float *>(d_v);
    A.end_state = static_cast<float *>(end_state);
    A.d_end = static_cast<float *>(d_end);
    A.status = status;
    mr::diff_tangent_kernel<float><<<mr::blocks_for(n), mr::kDiffBlock, 0, s>>>(A);
  } else {
    return fail(MR_ERR_INVALID_ARGUMENT, "precision must be 64 or 32");
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MR_OK : cuda_fail(e, "diff_tangent launch");
}

}  // extern "C"
