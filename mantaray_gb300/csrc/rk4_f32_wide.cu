// rk4_f32_wide.cu -- the single-scenario builds of the batched FP32 integrator
// for axes of more than 2^22 points (k2.cuh, locate), compiled like those of
// rk4_f32_one.cu.  The capped builds have 72 registers.  4.2 M x 9 nodes with a
// current on the grid, 1 M rays x 200 steps: blocks of 128 x 12 3.27 ms, x 4
// 4.77; through the uncapped scenario-table build 5.08 and 5.96.

#include "k2.cuh"
#include "kernels.h"

namespace mr {

template <int MODE>
static const void *wide_build(int build) {
  switch (build) {
    case 0: return reinterpret_cast<const void *>(&rk4_f32_kernel_1<MODE>);
    case 1:
    case 7: return reinterpret_cast<const void *>(&rk4_f32_kernel_1m<MODE>);
    case 5: return reinterpret_cast<const void *>(&rk4_f32_kernel_1s<MODE>);
    case 6:
    case 8: return reinterpret_cast<const void *>(&rk4_f32_kernel_1ms<MODE>);
    default: return reinterpret_cast<const void *>(&rk4_f32_kernel_2<MODE>);
  }
}

const void *rk4_f32_wide_function(int build, int same_grid) {
  return same_grid ? wide_build<10>(build) : wide_build<9>(build);
}

}  // namespace mr
