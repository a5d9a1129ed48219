// FP64 reciprocal square roots of the pair kernels.
#pragma once
#include <cuda_runtime.h>

namespace rtfmm_b200 {

// 1/sqrt(x) in FP64 from the hardware seed (one special-function op, 9.1e-7
// relative), and zero for x = 0; other x must be normal (pairs closer than
// 1e-154 are not supported).  The zero is made by the seed's words on the
// integer pipe: a comparison would take the FP64 pipe, which bounds every
// kernel that calls this.
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const int hi = __double2hiint(x);
  return __hiloint2double(hi ? __double2hiint(y) : 0, hi ? __double2loint(y) : 0);
}
// To full precision: with e = 1 - x y^2 the Taylor series of (1 - e)^(-1/2) to
// second order, y (1 + e/2 + 3 e^2/8) (Householder's method of third order;
// the remainder 5/16 e^3 is 2e-18): five operations, where two Newton steps
// take seven.
__device__ __forceinline__ double rsqrt_or_zero(double x) {
  const double y = rsqrt_seed(x);
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}
// Twice 1/sqrt(x) to 1.3e-12 (maximum against CUDA's rsqrt over 1e-30..1e30):
// one Newton step y (3 - x y^2), whose factor 1/2 the callers put into the
// charges, three operations instead of four.
__device__ __forceinline__ double rsqrt_twice(double x) {
  const double y = rsqrt_seed(x);
  return y * fma(-(x * y), y, 3.0);
}
// What the surface kernels use: FULL 1/sqrt(x), else 2/sqrt(x) with charges
// halved (kHalf, exact).
template <bool FULL>
__device__ __forceinline__ double rsqrt_surf(double x) {
  return FULL ? rsqrt_or_zero(x) : rsqrt_twice(x);
}

}  // namespace rtfmm_b200
