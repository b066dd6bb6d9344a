// qv_f64.cuh -- FP64 reciprocals and the straight-segment factor for the FP64
// pair sums.
//
// These sums are bound by FP64 issue (64 lanes per SM on sm_100), and the
// library's rsqrt and division carry range handling that positive, normal
// operands do not need.  Each function below starts from PTX's approximate
// FP64 instruction (rsqrt.approx.ftz.f64 / rcp.approx.ftz.f64, one MUFU) and
// takes one step of third order from the residual e of that estimate:
//   1/sqrt(a) = y (1 - e)^(-1/2) with e = 1 - a y^2,  series 1 + e/2 + 3 e^2/8
//   1/a       = y / (1 - e)      with e = 1 - a y,    series 1 + e + e^2
// An estimate good to 2^-18 or better leaves less than 2^-53 (tested against
// the library functions).  Operands: positive, normal, finite.
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ double rsqrt_pos(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-(a * y), y, 1.);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// n / a
__device__ __forceinline__ double div_pos(double n, double a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-a, y, 1.);
  const double ny = n * y;
  return fma(ny, fma(e, e, e), ny);
}

// Straight-segment factor f of u = f (R1 x s), s = R2 - R1
// (src/tree.f90:380-390): with A = |R1|^2, B = |R2|^2, d = R1.R2,
//   f = (|R1|+|R2|) / (|R1||R2| (|R1||R2| + d)) = (1/|R1| + 1/|R2|) q / (1 + d q),
// q = 1/(|R1||R2|).  For d > 0 (no cancellation in 1 + d q), A and B positive.
__device__ __forceinline__ double seg_f_pos(double A, double B, double d) {
  const double ra = rsqrt_pos(A), rb = rsqrt_pos(B);
  const double q = ra * rb;
  return div_pos((ra + rb) * q, fma(d, q, 1.));
}

// The same for any d: when d < 0 the sum |R1||R2| + d cancels and is taken from
// |R1 x s|^2 / (|R1||R2| - d) instead; c2 = |R1 x s|^2.  A point on the
// segment's line (c2 = 0) gets 0, as 4ac - b^2 = 0 is skipped in the reference
// (src/timestep.f90:476, 501).
__device__ __forceinline__ double seg_f_any(double A, double B, double d, double c2) {
  if (!(c2 > 0.) || !(B > 0.)) return c2 != c2 ? c2 : 0.;
  const double a = sqrt(A), b = sqrt(B), ab = a * b;
  const double e = d < 0. ? c2 / (ab - d) : ab + d;
  return (a + b) / (ab * e);
}
