// The IEEE quotient a / b of a divisor that many values share, from its
// correctly rounded reciprocal y = 1 / b: two corrections by exact residuals
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990). q = a*y is within two
// units of the quotient; the first correction leaves it within one, from where
// the second rounds it correctly. b is a permittivity or permeability, far from
// the ends of the exponent range; a near those ends (or not finite) takes the
// division itself, so that no residual underflows.
#pragma once

namespace fdtdb {

// whether quotient_of takes this dividend
__device__ __forceinline__ bool quotient_in_range(double a) {
  const unsigned hi = static_cast<unsigned>(__double2hiint(a)) & 0x7fffffffu;
  return hi - 0x08000000u < 0x70000000u || (hi | __double2loint(a)) == 0;  // 2^-895 <= |a| < 2^897, or zero
}

__device__ __forceinline__ double quotient_of(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  const double r = __fma_rn(__fma_rn(-q, b, a), y, q);
  return __fma_rn(__fma_rn(-r, b, a), y, r);
}

// the division itself, out of line: the loops that divide stay within the
// instruction cache
__device__ __noinline__ double plain_quotient(double a, double b) { return a / b; }

}  // namespace fdtdb
