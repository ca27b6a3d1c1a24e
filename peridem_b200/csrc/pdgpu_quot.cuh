// FP64 square roots and quotients of the bond loop.
//
// Root: the hardware's approximate reciprocal root, one third-order step
// (A. S. Householder, "The Numerical Treatment of a Single Nonlinear Equation",
// 1970), and the root corrected once by its exact residual.  Quotient: a y
// corrected once by its exact residual, with y ~ 1/b at hand.  (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990, for both corrections.)
//
// With y the rounded 1/b the quotient is the rounded one.  Where y is 1/sqrt(a) or
// its square (1.5 and 3 times 2^-53 off) the result before its last rounding is
// off by at most 12 * 2^-106 of itself, as the root's is: the rounded one, unless
// the exact result lies within 2^-49 of an ulp of the midpoint of two doubles,
// and then one of the two.  (A numerator below 2^-968 leaves a residual below the
// smallest normal number, which has fewer bits: the last one may differ there.)
#pragma once

namespace pdgpu {
namespace {

struct Root {
  double r, inv;  // sqrt(a), 1/sqrt(a)
};

// a inside [2^-900, 2^892]
__device__ __forceinline__ Root root_in_range(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  // 1/sqrt(a) = y (1 - e)^(-1/2) with e = 1 - a y^2, to second order in e
  const double e = __fma_rn(-(a * y), y, 1.0);
  y = __fma_rn(y * e, __fma_rn(e, 0.375, 0.5), y);
  const double r0 = a * y;
  return Root{__fma_rn(__fma_rn(-r0, r0, a), 0.5 * y, r0), y};
}
// any a: outside that range the plain root and division
__device__ __forceinline__ Root root(double a) {
  if ((unsigned)(__double2hiint(a) - 0x07b00000) < 0x70000000u) return root_in_range(a);
  const double r = sqrt(a);
  return Root{r, 1.0 / r};
}

// a / b, given y ~ 1/b
__device__ __forceinline__ double quot(double a, double b, double y) {
  const double q = a * y;
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// the same where the quotient may be infinite (its residual is not a number then)
__device__ __forceinline__ double quot_or_inf(double a, double b, double y) {
  const double q = a * y, c = __fma_rn(__fma_rn(-b, q, a), y, q);
  return c == c ? c : q;
}

}  // namespace
}  // namespace pdgpu
