// Branch-free FP64 square root and division for the bond passes.
//
// The correctly rounded __dsqrt_rn and __ddiv_rn each hold a branch for
// operands outside their fast range, which keeps the compiler from
// interleaving the bonds of a batch: the FP64 passes then waited on one
// dependent chain after another (issue slots 34 % busy, FP64 pipe 26 %). Here
// the range test is a value, so that a batch tests all its bonds at once and
// falls back to the built-in functions in one rare branch.
//
// Method: from an approximation y of 1/sqrt(a), the binomial series
//   1/sqrt(a) = y (1 - e)^(-1/2) = y (1 + e/2 + 3 e^2/8 + O(e^3)),  e = 1 - a y^2
// gives 1/sqrt(a) to within rounding (|e| < 2^-20, so e^3 < 2^-60), and the
// exact residuals a - g^2 and a - q b (one FMA each) round the root and the
// quotient correctly, as P. Markstein shows (IBM J. Res. Dev. 34(1), 1990).
#pragma once

#include <cuda_runtime.h>

namespace pdb {

struct RootD {
  double root, inv;  // sqrt(a); 1/sqrt(a) to about one unit in the last place
};

// a in [2^-900, 2^900] (root_in_range).
__device__ __forceinline__ RootD root_d(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-(a * y), y, 1.0);
  y = fma(fma(0.375, e, 0.5), y * e, y);
  const double g = a * y;
  RootD r;
  r.root = fma(fma(-g, g, a), 0.5 * y, g);
  r.inv = y;
  return r;
}

// False for zero, negative, tiny, huge and non-finite a.
__device__ __forceinline__ bool root_in_range(double a) {
  return (unsigned)(__double2hiint(a) - (123 << 20)) < (unsigned)(1800 << 20);
}

// 1/b rounded, from an approximation of it good to a few units in the last place.
__device__ __forceinline__ double recip_d(double b, double approx) { return fma(fma(-b, approx, 1.0), approx, approx); }

// a/b from rb = 1/b rounded.
__device__ __forceinline__ double quotient_d(double a, double b, double rb) {
  const double q = a * rb;
  return fma(fma(-q, b, a), rb, q);
}

}  // namespace pdb
