// hypot.hpp -- sqrt(a^2 + b^2) by the same operations and roundings on host and device.
//
// Borges' corrected form without fma ("An improved algorithm for hypot(a, b)", 2019): the
// rounded square root h of x^2 + y^2 less (h^2 - x^2 - y^2) / (2 h), whose numerator is a
// sum of differences that are exact or nearly so; below one ulp.  The tridiagonal solvers
// of host and device use it, so that neither depends on a C library's version of hypot.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define SADMRG_HD __host__ __device__ __forceinline__
#else
#define SADMRG_HD inline
#endif

namespace sadmrg {
namespace rn {   // one rounding each: the device compiler contracts plain a * b + c

#ifdef __CUDA_ARCH__
SADMRG_HD double add(double a, double b) { return __dadd_rn(a, b); }
SADMRG_HD double sub(double a, double b) { return __dsub_rn(a, b); }
SADMRG_HD double mul(double a, double b) { return __dmul_rn(a, b); }
SADMRG_HD double div(double a, double b) { return __ddiv_rn(a, b); }
SADMRG_HD double root(double a) { return __dsqrt_rn(a); }
#else
SADMRG_HD double add(double a, double b) { return a + b; }
SADMRG_HD double sub(double a, double b) { return a - b; }
SADMRG_HD double mul(double a, double b) { return a * b; }
SADMRG_HD double div(double a, double b) { return a / b; }
SADMRG_HD double root(double a) { return std::sqrt(a); }
#endif

// x >= y >= 0
SADMRG_HD double hypot_core(double x, double y) {
  const double h = root(add(mul(x, x), mul(y, y)));
  double num;
  if (h <= mul(2.0, y)) {
    const double t = sub(h, y);
    num = add(mul(x, sub(mul(2.0, t), x)), mul(sub(t, mul(2.0, sub(x, y))), t));
  } else {
    const double t = sub(h, x);
    num = add(mul(mul(2.0, t), sub(x, mul(2.0, y))), add(mul(sub(mul(4.0, t), y), y), mul(t, t)));
  }
  return sub(h, div(num, mul(2.0, h)));
}

// Numbers between these have squares, and products of their rounding errors (52 bits less),
// that neither overflow nor underflow.
constexpr double kHypotLo = 0x1p-300, kHypotHi = 0x1p300;

SADMRG_HD double hypot(double a, double b) {
  const double u = std::fabs(a), v = std::fabs(b), x = u < v ? v : u, y = u < v ? u : v;
  if (y >= kHypotLo && x <= kHypotHi) return hypot_core(x, y);
  if (add(x, y) == x || !(y <= x)) return add(x, y);   // y at most half an ulp of x; a NaN
  // with the larger scaled into [1, 2), exactly
  const int e = std::ilogb(x);
  return std::scalbn(hypot_core(std::scalbn(x, -e), std::scalbn(y, -e)), e);
}

}  // namespace rn
}  // namespace sadmrg
