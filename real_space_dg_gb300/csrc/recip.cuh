// 1 / x for chains of FP64 pivots, where a division's latency (447 cycles) is most of the chain.
#pragma once
#include <cuda_runtime.h>

namespace wg {

// The third-order iteration r (1 + e + e^2), e = 1 - x r, for the reciprocal (Altman's hyperpower method, Pacific Journal
// of Mathematics 10, 1960, for numbers; its error is e^3) from the instruction rcp.approx.ftz.f64, whose PTX
// specification gives about 20 bits: e^3 is below 2^-56, so the result is 1 / x with its one rounding and at most one unit of
// the last place off the correctly rounded quotient.  For 2^-1022 <= |x| <= 2^1022; beyond, where the instruction flushes:
// 0 for larger x, NaN for 0, subnormal numbers, infinities and NaN.
__device__ __forceinline__ double fast_rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

}  // namespace wg
