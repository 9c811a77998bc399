// packed.cuh -- two floats in one 64-bit register (f32x2): one instruction
// issues both halves' operation, at the rate of two scalar ones.  GB300's
// FP32 pipe does as many operations either way (39.4 T/s measured of fma and
// of fma.f32x2 pairs); what the packed form halves is issue slots.
//
// Each half rounds as the scalar operation does.  But ptxas contracts a
// packed product and a packed sum or difference of it into one FMA whatever
// -fmad and the rounding modifiers say (measured: every one of 20,000 random
// vadd(c, vmul(a, b)) equals fma(a, b, c)), so code that must not be
// contracted never feeds a vmul into a vadd or vsub, unless the product is
// exact: vmul_rn takes its place.
#pragma once

#include "bits.h"

namespace mr {

struct V { float x, y; };

#if defined(__CUDA_ARCH__)
#if defined(__CUDA_FTZ)
#define MR_F32X2 ".rn.ftz.f32x2 "
#else
#define MR_F32X2 ".rn.f32x2 "
#endif
#define MR_PACKED(name, op)                                                       \
  MR_HD V name(V a, V b) {                                                        \
    unsigned long long p, q, r;                                                   \
    V o;                                                                          \
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a.x), "f"(a.y));                  \
    asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(b.x), "f"(b.y));                  \
    asm(op MR_F32X2 "%0, %1, %2;" : "=l"(r) : "l"(p), "l"(q));                    \
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));                 \
    return o;                                                                     \
  }
MR_PACKED(vadd, "add")
MR_PACKED(vsub, "sub")
MR_PACKED(vmul, "mul")
#undef MR_PACKED
MR_HD V vfma(V a, V b, V c) {
  unsigned long long p, q, r, t;
  V o;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(c.x), "f"(c.y));
  asm("fma" MR_F32X2 "%0, %1, %2, %3;" : "=l"(t) : "l"(p), "l"(q), "l"(r));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(t));
  return o;
}
#undef MR_F32X2
#else
MR_HD V vadd(V a, V b) { return V{a.x + b.x, a.y + b.y}; }
MR_HD V vsub(V a, V b) { return V{a.x - b.x, a.y - b.y}; }
MR_HD V vmul(V a, V b) { return V{a.x * b.x, a.y * b.y}; }
MR_HD V vfma(V a, V b, V c) { return V{fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)}; }
#endif
MR_HD V both(float a) { return V{a, a}; }
// a b as two scalar products, which nothing contracts.
MR_HD V vmul_rn(V a, V b) {
#if defined(__CUDA_ARCH__)
  return V{__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)};
#else
  return V{a.x * b.x, a.y * b.y};
#endif
}
#if defined(__CUDACC__)
// a + b rounded toward minus infinity.
__device__ __forceinline__ V vadd_down(V a, V b) {
  unsigned long long p, q, r;
  V o;
  asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(q) : "f"(b.x), "f"(b.y));
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(p), "l"(q));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}
#endif

}  // namespace mr
