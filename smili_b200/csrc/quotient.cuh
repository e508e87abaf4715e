// Quotients by a divisor that many numerators share (host and device).
//
// Markstein's division with a reciprocal at hand (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Develop. 34 (1990) 111-119): with r = RN(1 / t) and q = RN(b r), the residual
// e = b - q t takes one fused multiply-add, and RN(q + e r) is the quotient.
// With u = 2^-53, q is within 2 u + u^2 of b / t, so q + e r is within 4 u^2 and
// the result within (1/2 + 2^-50) units in the last place, where the division
// guarantees 1/2.  That holds while r, q and e neither overflow nor leave the
// normal range: for |t| and |q| between 1e-140 and 1e140.  A zero numerator over
// such a t gives q itself, a zero; elsewhere the quotient is b / t.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define SMILI_HD __host__ __device__ __forceinline__
#define SMILI_HD_CALL __host__ __device__ __noinline__
#else
#define SMILI_HD inline
#define SMILI_HD_CALL inline
#endif

// 1 / t for div_by, or 0: divide
SMILI_HD double rcp_of(double t) {
  const double a = fabs(t);
  return a > 1e-140 && a < 1e140 ? 1.0 / t : 0.0;
}

// the rare case, out of line: five copies of the division's code cost a small
// solve more in instruction fetches than the range check itself
SMILI_HD_CALL double div_plain(double b, double t) { return b / t; }

// b / t from r = rcp_of(t): a third of the division's latency
SMILI_HD double div_by(double b, double t, double r) {
  const double q = b * r, a = fabs(q);
  if (a > 1e-140 && a < 1e140) return fma(fma(-q, t, b), r, q);
  return b == 0.0 && r != 0.0 ? q : div_plain(b, t);
}
