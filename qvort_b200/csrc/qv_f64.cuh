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

#include "qv_internal.cuh"

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

// f and its partial derivatives as a function of A = |R1|^2, w = R1.s and
// c = |s|^2 (B = A + 2 w + c, d = A + w): with m = |R1||R2|, e = m + d, S =
// |R1| + |R2|, f = S / (m e) and
//   fA = f (-((1/|R1| - 1/|R2|)^2 + 1/m) / 2 - ((A + B) / (2 m) + 1) / e)
//   fw = f (k - (A / m + 1) / e),   2 fc = f (k - (A / m) / e),
//   k  = 1 / (m + B) - 1 / B = -|R1| / (B S).
// The gradients of u = f (R1 x s) follow by the chain rule.
struct SegD {
  double f, fA, fw, fc2;  // fc2 = 2 df/dc
};
__device__ __forceinline__ SegD seg_d_of(double A, double B, double ra, double rb, double q,
                                         double ie, double iS) {
  SegD r;
  r.f = (ra + rb) * ie;
  const double k = -(A * ra) * (rb * rb) * iS;
  const double aq = A * q * ie, dr = ra - rb;
  r.fc2 = k - aq;
  r.fw = r.f * (r.fc2 - ie);
  r.fc2 *= r.f;
  r.fA = r.f * -fma(0.5, fma(dr, dr, q), fma(0.5 * (A + B), q, 1.) * ie);
  return r;
}
// d > 0
__device__ __forceinline__ SegD seg_d_pos(double A, double B, double d) {
  const double ra = rsqrt_pos(A), rb = rsqrt_pos(B), q = ra * rb;
  return seg_d_of(A, B, ra, rb, q, div_pos(q, fma(d, q, 1.)), div_pos(1., fma(A, ra, B * rb)));
}
// any d; c2 = |R1 x s|^2 (0: a point on the segment's line, no term)
__device__ __forceinline__ SegD seg_d_any(double A, double B, double d, double c2) {
  if (!(c2 > 0.) || !(B > 0.)) {
    const double z = c2 != c2 ? c2 : 0.;
    return SegD{z, z, z, z};
  }
  const double a = sqrt(A), b = sqrt(B), m = a * b;
  const double e = d < 0. ? c2 / (m - d) : m + d;
  return seg_d_of(A, B, 1. / a, 1. / b, 1. / m, 1. / e, 1. / (a + b));
}

// ------------------------------------------------------------ image sums
// Number of image shifts per axis (the reference's image loops,
// src/timestep.f90:235-257): PX x PY x PZ images, the unshifted one included.
template <int BC>
struct Img {
  static constexpr int PX = BC == QV_BC_PERIODIC ? 3 : 1;
  static constexpr int PY = (BC == QV_BC_PERIODIC || BC == QV_BC_OPENX) ? 3 : 1;
  static constexpr int PZ = BC == QV_BC_OPEN ? 1 : 3;
};

template <int P>
__device__ __forceinline__ void axis_shifts(double d, double L, double *r) {
  if (P == 3) {
    r[0] = d - L;
    r[1] = d;
    r[2] = d + L;
  } else {
    r[0] = d;
  }
}
template <int P>
__device__ __forceinline__ double least(const double *v) {
  return P == 3 ? fmin(fmin(v[0], v[1]), v[2]) : v[0];
}

// One source segment against one target in every image: R1 = x_j + shift - x_i
// and its square, per axis and shift.
template <int BC>
struct Seg64 {
  static constexpr int PX = Img<BC>::PX, PY = Img<BC>::PY, PZ = Img<BC>::PZ;
  double rx[PX], ry[PY], rz[PZ], px[PX], py[PY], pz[PZ];
  __device__ __forceinline__ Seg64(double dx, double dy, double dz, double L) {
    axis_shifts<PX>(dx, L, rx);
    axis_shifts<PY>(dy, L, ry);
    axis_shifts<PZ>(dz, L, rz);
#pragma unroll
    for (int e = 0; e < PX; e++) px[e] = rx[e] * rx[e];
#pragma unroll
    for (int e = 0; e < PY; e++) py[e] = ry[e] * ry[e];
#pragma unroll
    for (int e = 0; e < PZ; e++) pz[e] = rz[e] * rz[e];
  }
  // Whether |R1| > |s| in every image, so that R1.R2 >= |R1| (|R1| - |s|) > 0
  // (the _pos forms); the margin covers the rounding of both sides.
  __device__ __forceinline__ bool far(double c) const {
    return least<PX>(px) + least<PY>(py) + least<PZ>(pz) > 1.0001 * c;
  }
  // Adds the velocity terms of every image (the unshifted one unless skip_main)
  // to (ax, ay, az); s is the same in all of them, so f and f R1 are summed
  // over the images and the cross product is taken once.
  __device__ __forceinline__ void velocity(double sx, double sy, double sz, double c, double L,
                                           bool fast, bool skip_main, double &ax, double &ay,
                                           double &az) const {
    if (!fast) {
#pragma unroll 1
      for (int m = 0; m < PX * PY * PZ; m++) {
        if (skip_main && m == PX * PY * PZ / 2) continue;  // the middle one is unshifted
        double X, Y, Z;
        image(m, L, X, Y, Z);
        const double A = X * X + Y * Y + Z * Z, w = X * sx + Y * sy + Z * sz;
        const double cx = Y * sz - Z * sy, cy = Z * sx - X * sz, cz = X * sy - Y * sx;
        const double ex = X + sx, ey = Y + sy, ez = Z + sz;
        const double f =
            seg_f_any(A, ex * ex + ey * ey + ez * ez, A + w, cx * cx + cy * cy + cz * cz);
        ax += f * cx;
        ay += f * cy;
        az += f * cz;
      }
      return;
    }
    double fx[PX], fy[PY], fz[PZ];  // sum of f at each shift of an axis
#pragma unroll
    for (int k = 0; k < PX; k++) fx[k] = 0.;
#pragma unroll
    for (int k = 0; k < PY; k++) fy[k] = 0.;
#pragma unroll
    for (int k = 0; k < PZ; k++) fz[k] = 0.;
    // per-axis parts of A = |R1|^2 (p), d = R1.R2 = A + R1.s (g), B = |R2|^2 =
    // d + R1.s + |s|^2 (t)
    double gx[PX], tx[PX], gy[PY], ty[PY], gz[PZ], tz[PZ];
#pragma unroll
    for (int k = 0; k < PX; k++) { gx[k] = fma(rx[k], sx, px[k]); tx[k] = fma(rx[k], sx, gx[k] + c); }
#pragma unroll
    for (int k = 0; k < PY; k++) { gy[k] = fma(ry[k], sy, py[k]); ty[k] = fma(ry[k], sy, gy[k]); }
#pragma unroll
    for (int k = 0; k < PZ; k++) { gz[k] = fma(rz[k], sz, pz[k]); tz[k] = fma(rz[k], sz, gz[k]); }
#pragma unroll
    for (int a = 0; a < PX; a++) {
#pragma unroll
      for (int b = 0; b < PY; b++) {
        const double pxy = px[a] + py[b], gxy = gx[a] + gy[b], txy = tx[a] + ty[b];
        double row = 0.;
#pragma unroll
        for (int k = 0; k < PZ; k++) {
          const double f = seg_f_pos(pxy + pz[k], txy + tz[k], gxy + gz[k]);
          row += f;
          fz[k] += f;
        }
        fx[a] += row;
        fy[b] += row;
      }
    }
    double hx = 0., hy = 0., hz = 0.;
#pragma unroll
    for (int k = 0; k < PX; k++) hx = fma(fx[k], rx[k], hx);
#pragma unroll
    for (int k = 0; k < PY; k++) hy = fma(fy[k], ry[k], hy);
#pragma unroll
    for (int k = 0; k < PZ; k++) hz = fma(fz[k], rz[k], hz);
    ax += hy * sz - hz * sy;
    ay += hz * sx - hx * sz;
    az += hx * sy - hy * sx;
  }
  // R1 of image m (m = (a PY + b) PZ + k, shifts ascending)
  __device__ __forceinline__ void image(int m, double L, double &X, double &Y, double &Z) const {
    const int a = m / (PY * PZ), b = (m / PZ) % PY, k = m % PZ;
    X = PX == 3 ? rx[PX / 2] + (a - 1) * L : rx[0];
    Y = PY == 3 ? ry[PY / 2] + (b - 1) * L : ry[0];
    Z = PZ == 3 ? rz[PZ / 2] + (k - 1) * L : rz[0];
  }
};
