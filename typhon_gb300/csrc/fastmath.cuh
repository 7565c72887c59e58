// Reciprocal, reciprocal square root and square root for the fast mode (TY_MODE_FAST).
//
// GB300 issues FP64 at about 2 DFMA per SM per clock, and an IEEE FP64 division or square
// root costs about ten of them, so the fast kernels replace them with one Newton-Raphson
// step of third order in FP64, seeded by the hardware approximations of PTX
// (rcp.approx.ftz.f64 and rsqrt.approx.ftz.f64, which run on the special-function unit, not
// on the FP64 pipe; measured on GB300 to a relative error below 2^-19.9):
//
//   reciprocal of a:        e = 1 - a x,    x <- x (1 + e + e^2)             (3 DFMA)
//   reciprocal square root: e = 1 - a y^2,  y <- y (1 + e/2 + 3 e^2/8)       (5 FP64 ops)
//
// (Newton's iteration for f(x) = 1/x - a, and Halley's / the third-order Householder step
// for f(y) = 1/y^2 - a: the truncated binomial series of (1 - e)^(-1) and (1 - e)^(-1/2)).
// The remaining relative error is about e^3 ~ 2^-59, so the results are within a few units
// in the last place of the correctly rounded values (not always correctly rounded), which
// the fast mode's tolerance absorbs; ty_debug_fastmath measures them against CUDA's IEEE
// division and square root.  Inputs are positive normal numbers (densities, pressures, sums
// of squares): subnormal inputs are flushed to zero by the seeds.
#pragma once
#include <cuda_runtime.h>

namespace tyk {

__device__ __forceinline__ double rcp_seed(double a) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
  return r;
}

__device__ __forceinline__ double rsqrt_seed(double a) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a));
  return r;
}

// A double whose products and sums issue as fused multiply-adds: a b = fma(a, b, -0) and
// a + b = fma(a, 1, b), the same rounded values (signed zeros included).  On GB300 a DFMA with
// its three operands in registers issues every 64 clocks per SM quarter, a DMUL or DADD every 76
// (1.997 against 1.683 lanes per clock and SM), so kernels at the pipe's limit gain by it.  The
// constants come from memory so that they are registers to the assembler, not literals that it
// would fold back into DMUL and DADD.  Explicit fma() stays a DFMA; nothing is contracted.
static __device__ double g_f64_one = 1.0, g_f64_minus_zero = -0.0;
__device__ __forceinline__ double f64_one() {
  double r;
  asm("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(&g_f64_one));
  return r;
}
__device__ __forceinline__ double f64_minus_zero() {
  double r;
  asm("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(&g_f64_minus_zero));
  return r;
}
struct F64 {
  double v;
  F64() = default;
  __device__ __forceinline__ F64(double x) : v(x) {}
  friend __device__ __forceinline__ F64 operator*(F64 a, F64 b) { return ::fma(a.v, b.v, f64_minus_zero()); }
  friend __device__ __forceinline__ F64 operator+(F64 a, F64 b) { return ::fma(a.v, f64_one(), b.v); }
  friend __device__ __forceinline__ F64 operator-(F64 a, F64 b) { return ::fma(-b.v, f64_one(), a.v); }
  friend __device__ __forceinline__ F64 operator-(F64 a) { return -a.v; }
  friend __device__ __forceinline__ F64 fma(F64 a, F64 b, F64 c) { return ::fma(a.v, b.v, c.v); }
};

__device__ __forceinline__ double value(F64 a) { return a.v; }
__device__ __forceinline__ double value(double a) { return a; }

// 1/a: one third-order step from the hardware seed (3 DFMA).
__device__ __forceinline__ double rcp_nr(double a) {
  const double x = rcp_seed(a);
  const double e = fma(-a, x, 1.0);
  return fma(x, fma(e, e, e), x);
}

// 1/sqrt(a), a > 0: one third-order step from the hardware seed (5 FP64 operations).
__device__ __forceinline__ double rsqrt_nr(double a) {
  const double y = rsqrt_seed(a);
  const double e = fma(-a * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

__device__ __forceinline__ F64 rcp_nr(F64 a) {
  const F64 x = rcp_seed(a.v), e = fma(-a, x, f64_one());
  return fma(x, fma(e, e, e), x);
}
__device__ __forceinline__ F64 rsqrt_nr(F64 a) {
  const F64 y = rsqrt_seed(a.v), e = fma(-(a * y), y, f64_one());
  return fma(y * e, fma(F64(0.375), e, F64(0.5)), y);
}

// sqrt(a) = a / sqrt(a) for a > 0; 0 for a == 0 (the product would be 0 * inf) and for a < 0.
// The sign is read from the upper word: a comparison of doubles occupies the FP64 pipe.
__device__ __forceinline__ double sqrt_nr(double a) {
  const double r = a * rsqrt_nr(a);
  return __double2hiint(a) > 0 ? r : 0.0;
}

__device__ __forceinline__ F64 sqrt_nr(F64 a) {
  const F64 r = a * rsqrt_nr(a);
  return __double2hiint(a.v) > 0 ? r.v : 0.0;
}

// sqrt(a) as the library's for normal numbers: 0 for a == 0 (and subnormal a), NaN for a < 0.  For places
// where the root of a negative number has to show.
__device__ __forceinline__ F64 root_nr(F64 a) {
  const F64 r = a * rsqrt_nr(a);
  return ((unsigned)__double2hiint(a.v) << 1) < (2u << 20) ? 0.0 : r.v;
}
__device__ __forceinline__ double root_nr(double a) {
  const double r = a * rsqrt_nr(a);
  return ((unsigned)__double2hiint(a) << 1) < (2u << 20) ? 0.0 : r;
}

}  // namespace tyk
