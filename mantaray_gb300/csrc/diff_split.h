// diff_split.h -- launch interface of the FP64 differentiation kernels on
// float pairs (diff_split.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mr {

// One call's fields, rays and outputs (DiffArgs<double> in diff.cuh; that
// type is local to each unit, this one crosses).
struct DiffCall {
  const double *depth, *u, *v;
  int bnx, bny, cnx, cny;
  double bx0, by0, b_inv_dx, b_inv_dy;
  double cx0, cy0, c_inv_dx, c_inv_dy;
  int same_grid;
  int64_t n, steps, ck_every, n_ck;
  const double *x0, *y0, *kx0, *ky0;
  double dt;
  double *ckpt, *end_state;
  uint8_t *status;
  const double *grad_end;
  double *seg, *grad_state0, *grad_depth, *grad_u, *grad_v;
  const double *dstate0, *d_depth, *d_u, *d_v;
  double *d_end;
};

enum DiffForm : int { DIFF_FORWARD = 0, DIFF_ADJOINT = 1, DIFF_TANGENT = 2 };

// Runs the call on pairs; false (nothing queued) when they do not cover it or
// there is no memory for the records.  *err: the outcome of what was queued.
bool launch_diff_split(DiffForm form, const DiffCall &c, cudaStream_t stream, cudaError_t *err);

}  // namespace mr
