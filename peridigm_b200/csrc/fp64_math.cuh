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
// residuals a - g^2 and a - q b (one FMA each) round the root and the quotient
// correctly, as P. Markstein shows (IBM J. Res. Dev. 34(1), 1990), within these
// ranges, outside which the passes take the built-in functions:
//   root_in_range     the square: [2^-900, 2^900], so the root is in [2^-450, 2^450]
//   divisor_in_range  the divisor of a quotient: [2^-450, 2^450]
//   recip_in_range    the divisor of recip_d: not a significand of ones, whose
//                     reciprocal is so near the middle of two numbers that this
//                     step misses it (Markstein's exception)
// The numerator of a quotient is 0 or of a magnitude in [2^-500, 2^500). Above,
// a quotient that overflows, or an infinite numerator, gives NaN (inf - inf):
// an evaluation that ends with a force that is not finite is done again with
// the built-in functions alone. Below, from 2^-519 on, the residual underflows
// and the last bit may differ: terms of some 1e-160 and less, for which the
// passes do not look (a test of each numerator: 50 steps of 27x7x6 points 421 ->
// 495 us; of each row's sum: 20 steps of 131x97x21 points 12.5 -> 13.4 ms).
// tests/test_gpu_fp64_math.py compares the bits with the built-in functions'.
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

// True for a in [2^-450, 2^450].
__device__ __forceinline__ bool divisor_in_range(double a) {
  return (unsigned)(__double2hiint(a) - (573 << 20)) < (unsigned)(900 << 20);
}

// False for a significand of ones (and one in 2^32 others).
__device__ __forceinline__ bool recip_in_range(double b) { return __double2loint(b) != -1; }

// 1/b rounded, from 1/sqrt(b^2) as root_d gives it (recip_in_range).
__device__ __forceinline__ double recip_d(double b, double approx) { return fma(fma(-b, approx, 1.0), approx, approx); }

// a/b rounded, from rb = 1/b rounded (divisor_in_range; the numerator as above).
__device__ __forceinline__ double quotient_d(double a, double b, double rb) {
  const double q = a * rb;
  return fma(-fma(q, b, -a), rb, q);  // (the residual's sign keeps that of a zero)
}

}  // namespace pdb
