// Reciprocals and square roots for the FP64 film recursion.
//
// A division in IEEE double costs a long dependent instruction sequence; the
// film kernel needs several per order and layer.  Here 1/a is computed by
// Newton-Raphson iteration for the reciprocal, x <- x (2 - a x), which
// doubles the number of correct bits per step, seeded with the hardware's
// approximate double reciprocal (rcp.approx.ftz.f64): two steps give a result
// within a few ulps of 1/a (the film outputs agree with those of IEEE
// divisions to 1e-15 absolute).  Arguments whose magnitude is outside
// [2^-996, 2^996), and non-finite ones, take the IEEE division instead (the
// exponent field is compared: two integer operations for two of FP64).
#pragma once
#include "emu_cplx.cuh"

namespace emu {

// biased exponent of |a|
__device__ __forceinline__ unsigned exponent_of(double a) {
  return ((unsigned)__double2hiint(a) & 0x7fffffffu) >> 20;
}

__device__ __forceinline__ double rcp_nr(double a) {
  if (exponent_of(a) - 27u >= 1992u) return 1.0 / a;
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(a));
  double e = fma(-a, x, 1.0);
  x = fma(x, e, x);
  e = fma(-a, x, 1.0);
  x = fma(x, e, x);
  return x;
}

// 1 / z = conj(z) / |z|^2
__device__ __forceinline__ cd crcp_nr(cd z) {
  const double r = rcp_nr(fma(z.x, z.x, z.y * z.y));
  return cd{z.x * r, -z.y * r};
}

// 1/sqrt(a) for a normal positive a: Newton-Raphson for the reciprocal
// square root, y <- y (3/2 - a y^2 / 2), seeded with the hardware's
// approximate double reciprocal square root (rsqrt.approx.ftz.f64); two
// steps, as for rcp_nr.
__device__ __forceinline__ double rsqrt_nr(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double ha = 0.5 * a;
  double e = fma(-ha * y, y, 0.5);
  y = fma(y, e, y);
  e = fma(-ha * y, y, 0.5);
  y = fma(y, e, y);
  return y;
}

// Principal square root for k_z (C99 csqrt branch rules, Kahan's form
// t = sqrt((|x| + |z|)/2)) from two reciprocal square roots: |z| = q / sqrt(q)
// with q = |z|^2, t = s / sqrt(s) and 1/(2t) = 1/(2 sqrt(s)) with
// s = (|x| + |z|)/2.  Where |z|^2 would leave the normal range (and for zero
// or non-finite z) it takes the IEEE form csqrt_p.  Both give exact zeros
// and exactly real or exactly imaginary results for the same arguments.
__device__ __forceinline__ cd csqrt_k(cd z) {
  const double ax = fabs(z.x), ay = fabs(z.y);
  // the larger part within [2^-498, 2^498)
  if (max(exponent_of(ax), exponent_of(ay)) - 525u >= 996u) return csqrt_p(z);
  if (ay == 0.0) {
    // a real argument: one root and one correction step, for the k_z of air and of
    // lossless layers
    const double r = rsqrt_nr(ax);
    double t = ax * r;
    t = fma(fma(-t, t, ax), 0.5 * r, t);
    return z.x >= 0.0 ? cd{t, z.y} : cd{0.0, copysign(t, z.y)};
  }
  const double q = fma(z.x, z.x, z.y * z.y);
  const double h = q * rsqrt_nr(q);
  const double sh = 0.5 * (ax + h);
  const double r = rsqrt_nr(sh);
  const double t = sh * r;
  const double hr = 0.5 * r;
  if (z.x >= 0.0) return cd{t, z.y * hr};
  return cd{ay * hr, copysign(t, z.y)};
}

// csqrt_p(z).y == 0 (the order propagates) decided from z itself: the
// principal root is real exactly when z is real and not negative.
__device__ __forceinline__ bool sqrt_is_real(cd z) { return z.y == 0.0 && z.x >= 0.0; }

}  // namespace emu
