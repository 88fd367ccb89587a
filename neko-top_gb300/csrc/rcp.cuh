// The FP64 reciprocal of the optimiser's kernels (mma.cu).
#pragma once

namespace ntg {

// 1/x by the third-order iteration r (1 + e + e^2), e = 1 - x r (Householder),
// from the hardware's approximation r0: e0 < 2^-19 leaves e0^3 < 2^-57, the
// result within an ulp.  The FP64 pipe (2 operations per clock and SM) bounds
// these kernels; this takes three of them, a division about ten.
__device__ __forceinline__ double rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(fma(e, e, e), r, r);
}

}  // namespace ntg
