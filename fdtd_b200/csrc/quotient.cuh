// The IEEE quotient a / b of a divisor that many values share, from its
// correctly rounded reciprocal y = 1 / b: two corrections by exact residuals
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34, 1990). q = a*y is within two
// units of the quotient; the first correction leaves it within one, from where
// the second rounds it correctly. A dividend or divisor near the ends of the
// exponent range (or not finite) takes the division itself, so that no residual
// underflows or overflows, and so does -0, whose sign the residuals lose.
#pragma once

namespace fdtdb {

// the reciprocal that quotient_of takes, zero for a divisor out of its range
__host__ __device__ inline double quotient_reciprocal(double b) { return b >= 0x1p-100 && b <= 0x1p100 ? 1.0 / b : 0.0; }
__device__ __forceinline__ bool quotient_by(double y) { return __double2hiint(y) != 0; }

// whether quotient_of takes this dividend
__device__ __forceinline__ bool quotient_in_range(double a) {
  const unsigned hi = static_cast<unsigned>(__double2hiint(a));
  return (hi & 0x7fffffffu) - 0x08000000u < 0x70000000u || (hi | __double2loint(a)) == 0;  // 2^-895 <= |a| < 2^897, or +0
}

__device__ __forceinline__ double quotient_of(double a, double b, double y) {
  const double q = __dmul_rn(a, y);
  const double r = __fma_rn(__fma_rn(-q, b, a), y, q);
  return __fma_rn(__fma_rn(-r, b, a), y, r);
}

// the division itself, out of line: the loops that divide stay within the
// instruction cache
static __device__ __noinline__ double plain_quotient(double a, double b) { return a / b; }

}  // namespace fdtdb
