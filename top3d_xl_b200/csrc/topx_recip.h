// Refinement of a reciprocal approximation, for the device code and for a host program that checks it.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define TOPX_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TOPX_HOST_DEVICE inline
#endif

namespace topx {

// 1/v from an approximation x of it: with e = 1 - v x the geometric series 1/v = x / (1 - e) = x (1 + e + e^2 + e^3 + ...),
// formed to e^3 as x + (x e) (1 + e + e^2).  1 + e is 2 - v x, beside e, so three operations depend on one another,
// as many as for the series to e^2 and one fewer than two Newton-Raphson steps take for the same remainder e^4: with the 20
// bits of the hardware's approximation 2^-80.  The error left is the last operation's rounding, 2^-53 at most, as for
// two Newton-Raphson steps (the series to e^2 leaves 1.006 x 2^-53).
TOPX_HOST_DEVICE double recip_series(double v, double x) {
  const double e = fma(-v, x, 1.0), e1 = fma(-v, x, 2.0);
  return fma(x * e, fma(e, e, e1), x);
}

}  // namespace topx
