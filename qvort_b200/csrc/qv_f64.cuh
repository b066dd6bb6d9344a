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
// c = |s|^2 (B = A + 2 w + c, d = A + w): with a = |R1|, b = |R2|, m = a b, q =
// 1 / m, e = m + d and g = f / e (1 / m + 1 / B and the like written through the
// reciprocals at hand; the sum a + b in f = (a + b) / (m e) cancels from the
// derivatives of its logarithm)
//   2 fA = -(f ((1/a - 1/b)^2 + q) + g ((A + B) q + 2))
//   2 fc = -(1/b^3 + f A q) / e,   fw = 2 fc - g.
// The gradients of u = f (R1 x s) follow by the chain rule.
struct SegD {
  double f, fA2, fw, fc2;  // f, 2 df/dA, df/dw, 2 df/dc
};
__device__ __forceinline__ SegD seg_d_of(double A, double B, double ra, double rb, double q,
                                         double ie) {
  SegD r;
  r.f = (ra + rb) * ie;
  const double g = r.f * ie, dr = ra - rb;
  r.fc2 = -ie * fma(rb * rb, rb, r.f * (A * q));
  r.fw = r.fc2 - g;
  r.fA2 = -fma(r.f, fma(dr, dr, q), g * fma(A + B, q, 2.));
  return r;
}
// d > 0
__device__ __forceinline__ SegD seg_d_pos(double A, double B, double d) {
  const double ra = rsqrt_pos(A), rb = rsqrt_pos(B), q = ra * rb;
  return seg_d_of(A, B, ra, rb, q, div_pos(q, fma(d, q, 1.)));
}
// any d; c2 = |R1 x s|^2 (0: a point on the segment's line, no term)
__device__ __forceinline__ SegD seg_d_any(double A, double B, double d, double c2) {
  if (!(c2 > 0.) || !(B > 0.)) {
    const double z = c2 != c2 ? c2 : 0.;
    return SegD{z, z, z, z};
  }
  const double a = sqrt(A), b = sqrt(B), m = a * b;
  const double e = d < 0. ? c2 / (m - d) : m + d;
  return seg_d_of(A, B, 1. / a, 1. / b, 1. / m, 1. / e);
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

// One source segment against one target in every image.  Per axis and shift:
// R1 = x_j + shift - x_i (r) and the parts of |R1|^2 (p) and R1.R2 (g); the sum
// over the axes gives an image's value.
template <int BC>
struct Seg64 {
  static constexpr int PX = Img<BC>::PX, PY = Img<BC>::PY, PZ = Img<BC>::PZ;
  static constexpr int NI = PX * PY * PZ;
  double sx, sy, sz, c;  // segment vector s and |s|^2
  double rx[PX], ry[PY], rz[PZ], px[PX], py[PY], pz[PZ], gx[PX], gy[PY], gz[PZ];
  __device__ __forceinline__ Seg64(double dx, double dy, double dz, double sx_, double sy_,
                                   double sz_, double c_, double L)
      : sx(sx_), sy(sy_), sz(sz_), c(c_) {
    axis_shifts<PX>(dx, L, rx);
    axis_shifts<PY>(dy, L, ry);
    axis_shifts<PZ>(dz, L, rz);
#pragma unroll
    for (int e = 0; e < PX; e++) { px[e] = rx[e] * rx[e]; gx[e] = fma(rx[e], sx, px[e]); }
#pragma unroll
    for (int e = 0; e < PY; e++) { py[e] = ry[e] * ry[e]; gy[e] = fma(ry[e], sy, py[e]); }
#pragma unroll
    for (int e = 0; e < PZ; e++) { pz[e] = rz[e] * rz[e]; gz[e] = fma(rz[e], sz, pz[e]); }
  }
  // Whether R1.R2 > |s|^2 / 16 in every image that is summed: the _pos forms
  // hold there, and |R2|^2 = R1.R2 + R1.s + |s|^2 keeps its digits (both ends
  // lie well off the target).  Every point's own neighbours pass, so only
  // points about to reconnect take the general form.  The least R1.R2 over
  // the images is the sum of the axes' least parts.  skip_main (the point's
  // own segment): the other images lie a box side away.
  __device__ __forceinline__ bool far(bool skip_main, double L) const {
    if (skip_main) return c < 0.25 * L * L;
    return least<PX>(gx) + least<PY>(gy) + least<PZ>(gz) > 0.0625 * c;
  }
  // R1 of image m (m = (a PY + b) PZ + k, shifts ascending)
  __device__ __forceinline__ void image(int m, double L, double &X, double &Y, double &Z) const {
    const int a = m / (PY * PZ), b = (m / PZ) % PY, k = m % PZ;
    X = PX == 3 ? rx[PX / 2] + (a - 1) * L : rx[0];
    Y = PY == 3 ? ry[PY / 2] + (b - 1) * L : ry[0];
    Z = PZ == 3 ? rz[PZ / 2] + (k - 1) * L : rz[0];
  }
  // Adds the velocity terms of every image (the unshifted one unless skip_main)
  // to (ax, ay, az).  s is the same in all of them, so f and f R1 are summed
  // over the images -- sum f R1 per axis is the sum over its shifts of (R1
  // component) x (sum of f at that shift) -- and the cross product is taken
  // once.  fast: far() holds.
  __device__ __forceinline__ void velocity(double L, bool fast, bool skip_main, double &ax,
                                           double &ay, double &az) const {
    if (!fast) {
#pragma unroll 1
      for (int m = 0; m < NI; m++) {
        if (skip_main && m == NI / 2) continue;  // the middle one is unshifted
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
    double tx[PX], ty[PY], tz[PZ];  // parts of |R2|^2 = R1.R2 + R1.s + |s|^2
#pragma unroll
    for (int k = 0; k < PX; k++) { fx[k] = 0.; tx[k] = fma(rx[k], sx, gx[k] + c); }
#pragma unroll
    for (int k = 0; k < PY; k++) { fy[k] = 0.; ty[k] = fma(ry[k], sy, gy[k]); }
#pragma unroll
    for (int k = 0; k < PZ; k++) { fz[k] = 0.; tz[k] = fma(rz[k], sz, gz[k]); }
#pragma unroll
    for (int a = 0; a < PX; a++) {
#pragma unroll
      for (int b = 0; b < PY; b++) {
        const double pxy = px[a] + py[b], gxy = gx[a] + gy[b], txy = tx[a] + ty[b];
        double row = 0.;
#pragma unroll
        for (int k = 0; k < PZ; k++) {
          double A = pxy + pz[k], B = txy + tz[k], d = gxy + gz[k];
          const bool own = skip_main && (a * PY + b) * PZ + k == NI / 2;
          if (own) A = B = d = 1.;
          double f = seg_f_pos(A, B, d);
          if (own) f = 0.;
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
  // Whether some image may have its target exactly on the segment's line
  // (R1 x s = 0): those terms' gradients are left out.
  __device__ __forceinline__ bool on_line() const {
    bool z = false;
#pragma unroll
    for (int a = 0; a < PX; a++)
#pragma unroll
      for (int b = 0; b < PY; b++) z |= rx[a] * sy - ry[b] * sx == 0.;
    if (!z) return false;
    z = false;
#pragma unroll
    for (int b = 0; b < PY; b++)
#pragma unroll
      for (int k = 0; k < PZ; k++) z |= ry[b] * sz - rz[k] * sy == 0.;
    if (!z) return false;
    z = false;
#pragma unroll
    for (int a = 0; a < PX; a++)
#pragma unroll
      for (int k = 0; k < PZ; k++) z |= rz[k] * sx - rx[a] * sz == 0.;
    return z;
  }
  // For an upstream g, the gradient of g . sum over images of f (R1 x s): dR
  // with respect to x_j at fixed s (minus the target's), dS with respect to s.
  // With h = s x g, Q = g.(R1 x s) = R1.h, alpha = 2 Q fA, beta = Q fw:
  //   dR = h sum f + sum alpha R1 + s sum beta
  //   dS = g x sum f R1 + sum beta R1 + s sum Q 2 fc
  // fast: far() holds and on_line() does not.
  __device__ __forceinline__ void gradient(double ux, double uy, double uz, double L, bool fast,
                                           bool skip_main, double *dR, double *dS) const {
    const double hx = sy * uz - sz * uy, hy = sz * ux - sx * uz, hz = sx * uy - sy * ux;
    double f0 = 0., b0 = 0., c0 = 0.;
    double fX = 0., fY = 0., fZ = 0., aX = 0., aY = 0., aZ = 0., bX = 0., bY = 0., bZ = 0.;
    if (fast) {
      double ty[PY], tz[PZ], qy[PY], qz[PZ];
#pragma unroll
      for (int k = 0; k < PY; k++) { ty[k] = fma(ry[k], sy, gy[k]); qy[k] = ry[k] * hy; }
#pragma unroll
      for (int k = 0; k < PZ; k++) { tz[k] = fma(rz[k], sz, gz[k]); qz[k] = rz[k] * hz; }
#pragma unroll 1  // a third of the code and registers: three blocks per SM
      for (int a = 0; a < PX; a++) {
        const double xa = PX == 3 ? rx[PX / 2] + (a - 1) * L : rx[0], pa = xa * xa,
                     ga = fma(xa, sx, pa), ta = fma(xa, sx, ga + c), qa = xa * hx;
        double fa = 0., aa = 0., ba = 0.;  // sums over the shifts (b, k) of this a
#pragma unroll
        for (int b = 0; b < PY; b++) {
          const double pxy = pa + py[b], gxy = ga + gy[b], txy = ta + ty[b],
                       qxy = qa + qy[b];
          double fb = 0., ab = 0., bb = 0.;
#pragma unroll
          for (int k = 0; k < PZ; k++) {
            double A = pxy + pz[k], B = txy + tz[k], d = gxy + gz[k];
            double Q = qxy + qz[k];
            const bool own = skip_main && (a * PY + b) * PZ + k == NI / 2;
            if (own) A = B = d = 1.;
            SegD t = seg_d_pos(A, B, d);
            if (own) t.f = Q = 0.;
            const double al = Q * t.fA2, be = Q * t.fw;
            c0 = fma(Q, t.fc2, c0);
            fb += t.f; ab += al; bb += be;
            fZ = fma(t.f, rz[k], fZ);
            aZ = fma(al, rz[k], aZ);
            bZ = fma(be, rz[k], bZ);
          }
          fa += fb; aa += ab; ba += bb;
          fY = fma(fb, ry[b], fY);
          aY = fma(ab, ry[b], aY);
          bY = fma(bb, ry[b], bY);
        }
        f0 += fa; b0 += ba;
        fX = fma(fa, xa, fX);
        aX = fma(aa, xa, aX);
        bX = fma(ba, xa, bX);
      }
    } else {
#pragma unroll 1
      for (int m = 0; m < NI; m++) {
        if (skip_main && m == NI / 2) continue;
        double X, Y, Z;
        image(m, L, X, Y, Z);
        const double A = X * X + Y * Y + Z * Z, w = X * sx + Y * sy + Z * sz;
        const double cx = Y * sz - Z * sy, cy = Z * sx - X * sz, cz = X * sy - Y * sx;
        const double ex = X + sx, ey = Y + sy, ez = Z + sz;
        const SegD t =
            seg_d_any(A, ex * ex + ey * ey + ez * ez, A + w, cx * cx + cy * cy + cz * cz);
        const double Q = X * hx + Y * hy + Z * hz, al = Q * t.fA2, be = Q * t.fw;
        f0 += t.f; b0 += be; c0 += Q * t.fc2;
        fX += t.f * X; fY += t.f * Y; fZ += t.f * Z;
        aX += al * X; aY += al * Y; aZ += al * Z;
        bX += be * X; bY += be * Y; bZ += be * Z;
      }
    }
    dR[0] = fma(hx, f0, fma(sx, b0, aX));
    dR[1] = fma(hy, f0, fma(sy, b0, aY));
    dR[2] = fma(hz, f0, fma(sz, b0, aZ));
    dS[0] = fma(sx, c0, bX) + (uy * fZ - uz * fY);
    dS[1] = fma(sy, c0, bY) + (uz * fX - ux * fZ);
    dS[2] = fma(sz, c0, bZ) + (ux * fY - uy * fX);
  }
};
