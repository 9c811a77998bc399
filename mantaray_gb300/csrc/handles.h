// handles.h -- the library's handle types and error helpers (internal).
#pragma once

#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "fields.h"

namespace mr {

// A gridded field's axes as f32, on the host, where it has records (SplitGrid).
struct SplitAxes {
  std::vector<float> x, y;
  float sp_x = 0.0f, sp_y = 0.0f;
  bool affine = false;
};

// Records are built with the handle (the traces themselves allocate nothing)
// and stay with it, so they may take an eighth of the free memory at most: what
// a program allocates after its handles, such as a batch's cells, has room as
// before.  Up to kSplitSmallBytes is not looked at.
constexpr size_t kSplitSmallBytes = size_t(32) << 20;
inline bool split_records_fit(size_t bytes, size_t free_bytes) {
  return bytes <= kSplitSmallBytes || bytes <= free_bytes / 8;
}

}  // namespace mr

struct mr_bathymetry {
  mr::BathyDev dev{};
  int device = 0;
  bool one_point_axis = false;  // the reference panics on its first lookup
  std::vector<void *> mem;      // device allocations owned by the handle
  mr::SplitAxes axes;
};

struct mr_current {
  mr::CurrentDev dev{};
  int device = 0;
  bool one_point_axis = false;
  std::vector<void *> mem;
  mr::SplitAxes axes;
};

namespace mr {

extern thread_local std::string g_last_error;

// Records a formatted message for mr_last_error() and returns `code`.
int fail(int code, const char *fmt, ...);
// MR_ERR_CUDA / MR_ERR_OUT_OF_MEMORY with the CUDA error's name.
int cuda_fail(cudaError_t e, const char *what);

// Makes `device` current for the lifetime of the guard.
class DeviceGuard {
 public:
  explicit DeviceGuard(int device) {
    ok_ = cudaGetDevice(&prev_) == cudaSuccess;
    if (ok_ && prev_ != device) ok_ = cudaSetDevice(device) == cudaSuccess;
    switched_ = ok_ && prev_ != device;
  }
  ~DeviceGuard() {
    if (switched_) cudaSetDevice(prev_);
  }
  bool ok() const { return ok_; }

 private:
  int prev_ = 0;
  bool ok_ = false;
  bool switched_ = false;
};

}  // namespace mr

#define MR_CUDA(call)                                           \
  do {                                                          \
    cudaError_t e_ = (call);                                    \
    if (e_ != cudaSuccess) return mr::cuda_fail(e_, #call);     \
  } while (0)
