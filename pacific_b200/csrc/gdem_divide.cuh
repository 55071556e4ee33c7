// gdem_divide.cuh -- FP64 division by a constant whose reciprocal is known.
#pragma once
#include <cmath>
#include <cuda_runtime.h>

namespace gdem {

// a / b, correctly rounded, for a divisor b > 0 whose correctly rounded
// reciprocal is rb: the quotient a rb corrected twice by its exact FMA
// remainder (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990: a faithful quotient
// corrected once with a correctly rounded reciprocal is the rounded one; the
// first correction makes it faithful).  Outside 1e-200 .. 1e200, where a
// remainder could lose bits, and without a reciprocal (rb = 0), a plain
// division.  What it is for: the FP64 leapfrog was bound by the issue of its
// 19 divisions per particle, 18 of them by constants of the class (256,000
// spheres: move kernel 43.1 us with them, 22.8 us so).
__host__ __device__ __forceinline__ double divideBy(double a, double b, double rb) {
  const double q0 = a * rb;
  if (a == 0. && rb > 0.) return q0;   // (the zero keeps its sign)
  const double m = fabs(a);
  if (!(m >= 1.e-200 && m <= 1.e200 && rb > 0.)) return a / b;
  const double q1 = fma(fma(-b, q0, a), rb, q0);
  return fma(fma(-b, q1, a), rb, q1);
}

// The reciprocal divideBy takes for b; none (0) for a divisor so large or
// small that a quotient or remainder could leave the normal range.
inline double reciprocalFor(double b) { return b >= 1.e-100 && b <= 1.e100 ? 1. / b : 0.; }

}  // namespace gdem
