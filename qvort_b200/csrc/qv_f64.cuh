// qv_f64.cuh -- FP64 reciprocals and the straight-segment factor for the FP64
// pair sums.
//
// These sums are bound by FP64 issue (64 lanes per SM on sm_100), and the
// library's rsqrt and division carry range handling that positive, normal
// operands do not need.  Each function below starts from PTX's approximate
// FP64 instruction (rsqrt.approx.ftz.f64 / rcp.approx.ftz.f64, one MUFU; the low 32
// bits of what they return are zeros) and takes one step of Householder's third
// order from the residual e of that estimate:
//   1/sqrt(a) = y (1 - e)^(-1/2) with e = 1 - a y^2,  series 1 + e/2 + 3 e^2/8
//   1/a       = y / (1 - e)      with e = 1 - a y,    series 1 + e + e^2
// The square of a 21-bit estimate is exact, so e of the root is rounded once, and
// what is left out (5 e^3/16, e^3) is below 0.2 2^-53 for an estimate good to
// 2^-19: the root's error is that of one rounding, 1.2 2^-53 at most, the quotient's
// that of two, 2.1 2^-53.  qv_test_f64 holds them to these bounds.  Operands:
// positive, normal, finite.
#pragma once
#include <cuda_runtime.h>

#include "qv_internal.cuh"

__device__ __forceinline__ double rsqrt_pos(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-a, y * y, 1.);
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

// f and its partial derivatives as a function of A = |R1|^2, B = |R2|^2 and d =
// R1.R2: with a = |R1|, b = |R2| and e = a b + d, f = (a + b) / (a b e) and
//   2 fA = -(1/a^2 + f b) / (a e),   2 fB = -(1/b^2 + f a) / (b e),   fd = -f / e,
// sums of one sign, so a target near either end keeps every digit, as long as R2
// and the products above are formed from R2 itself.  (The derivatives by R1 and
// s, B = |R1|^2 + 2 R1.s + |s|^2, save a vector sum but cancel near R2's end: 5e-14
// of the gradient at 0.07 |s| from it.)  The gradients of u = f (R1 x R2) follow by
// the chain rule.
struct SegD {
  double f, fA2, fB2, fd;  // f, and Q times 2 df/dA, 2 df/dB, df/dd
};
__device__ __forceinline__ SegD seg_d_of(double A, double B, double ra, double rb, double ie,
                                         double Q) {
  SegD r;
  r.f = (ra + rb) * ie;
  const double qe = -Q * ie;
  r.fA2 = (qe * ra) * fma(ra, ra, r.f * (B * rb));
  r.fB2 = (qe * rb) * fma(rb, rb, r.f * (A * ra));
  r.fd = qe * r.f;
  return r;
}
// d > 0
__device__ __forceinline__ SegD seg_d_pos(double A, double B, double d, double Q) {
  const double ra = rsqrt_pos(A), rb = rsqrt_pos(B), q = ra * rb;
  return seg_d_of(A, B, ra, rb, div_pos(q, fma(d, q, 1.)), Q);
}
// any d; c2 = |R1 x s|^2 (0: a point on the segment's line, no term)
__device__ __forceinline__ SegD seg_d_any(double A, double B, double d, double c2, double Q) {
  if (!(c2 > 0.) || !(B > 0.)) {
    const double z = c2 != c2 ? c2 : 0.;
    return SegD{z, z, z, z};
  }
  const double a = sqrt(A), b = sqrt(B), m = a * b;
  const double e = d < 0. ? c2 / (m - d) : m + d;
  return seg_d_of(A, B, 1. / a, 1. / b, 1. / e, Q);
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
// R1 = x_j + shift - x_i (r), R2 = ghost_j + shift - x_i (e) and the parts of
// |R1|^2 (p), |R2|^2 (t) and R1.R2 (g); the sum over the axes gives an image's value.
template <int BC>
struct Seg64 {
  static constexpr int PX = Img<BC>::PX, PY = Img<BC>::PY, PZ = Img<BC>::PZ;
  static constexpr int NI = PX * PY * PZ;
  double sx, sy, sz, c;  // segment vector s and |s|^2
  double rx[PX], ry[PY], rz[PZ], ex[PX], ey[PY], ez[PZ];
  double px[PX], py[PY], pz[PZ], tx[PX], ty[PY], tz[PZ], gx[PX], gy[PY], gz[PZ];
  // (dx, dy, dz) = R1 and (fx, fy, fz) = R2 of the unshifted image
  __device__ __forceinline__ Seg64(double dx, double dy, double dz, double fx, double fy, double fz,
                                   double sx_, double sy_, double sz_, double c_, double L)
      : sx(sx_), sy(sy_), sz(sz_), c(c_) {
    axis<PX>(dx, fx, L, rx, ex, px, tx, gx);
    axis<PY>(dy, fy, L, ry, ey, py, ty, gy);
    axis<PZ>(dz, fz, L, rz, ez, pz, tz, gz);
  }
  template <int P>
  __device__ __forceinline__ static void axis(double d, double f, double L, double *r, double *e,
                                              double *p, double *t, double *g) {
    axis_shifts<P>(d, L, r);
    axis_shifts<P>(f, L, e);
#pragma unroll
    for (int k = 0; k < P; k++) { p[k] = r[k] * r[k]; t[k] = e[k] * e[k]; g[k] = r[k] * e[k]; }
  }
  // Whether R1.R2 > |s|^2 / 16 in every image that is summed: the _pos forms
  // hold there (both ends lie off the target, by 0.06 |s| at least).  Every
  // point's own neighbours pass, so only points about to reconnect take the
  // general form.  The least R1.R2 over the images is the sum of the axes' least
  // parts.  skip_main (the point's own segment): the other images lie a box side
  // away.
  __device__ __forceinline__ bool far(bool skip_main, double L) const {
    if (skip_main) return c < 0.25 * L * L;
    return least<PX>(gx) + least<PY>(gy) + least<PZ>(gz) > 0.0625 * c;
  }
  // R1 and R2 of image m (m = (a PY + b) PZ + k, shifts ascending)
  __device__ __forceinline__ void image(int m, double L, double *R1, double *R2) const {
    const double X = PX == 3 ? (m / (PY * PZ) - 1) * L : 0.,
                 Y = PY == 3 ? ((m / PZ) % PY - 1) * L : 0., Z = PZ == 3 ? (m % PZ - 1) * L : 0.;
    R1[0] = rx[PX / 2] + X; R1[1] = ry[PY / 2] + Y; R1[2] = rz[PZ / 2] + Z;
    R2[0] = ex[PX / 2] + X; R2[1] = ey[PY / 2] + Y; R2[2] = ez[PZ / 2] + Z;
  }
  // A, B, d and R1 x s = R2 x s of an image, the product from the nearer end: the
  // other one's cancels beside the segment's line.  The target is on that line
  // where R1 x s vanishes.
  __device__ __forceinline__ void image_term(const double *R1, const double *R2, double &A,
                                             double &B, double &d, double *cr) const {
    A = R1[0] * R1[0] + R1[1] * R1[1] + R1[2] * R1[2];
    B = R2[0] * R2[0] + R2[1] * R2[1] + R2[2] * R2[2];
    d = R1[0] * R2[0] + R1[1] * R2[1] + R1[2] * R2[2];
    cross_s(R1, cr);
    if (B < A && (cr[0] != 0. || cr[1] != 0. || cr[2] != 0.)) {
      double q[3];
      cross_s(R2, q);
      if (q[0] != 0. || q[1] != 0. || q[2] != 0.) { cr[0] = q[0]; cr[1] = q[1]; cr[2] = q[2]; }
    }
  }
  __device__ __forceinline__ void cross_s(const double *R, double *cr) const {
    cr[0] = R[1] * sz - R[2] * sy;
    cr[1] = R[2] * sx - R[0] * sz;
    cr[2] = R[0] * sy - R[1] * sx;
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
        if (skip_main && m == NI / 2) continue;
        double R1[3], R2[3], cr[3], A, B, d;
        image(m, L, R1, R2);
        image_term(R1, R2, A, B, d, cr);
        const double f = seg_f_any(A, B, d, cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2]);
        ax += f * cr[0];
        ay += f * cr[1];
        az += f * cr[2];
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
  // For an upstream g, the gradient of g . sum over images of f (R1 x R2): dR
  // with respect to x_j at fixed s (minus the target's), dS with respect to s.
  // With h = s x g, Q = g.(R1 x R2) = R1.h = R2.h, alpha = 2 Q fA, beta = 2 Q fB and
  // gamma = Q fd:
  //   dS = g x sum f R1 + sum beta R2 + sum gamma R1
  //   dR = h sum f + sum alpha R1 + sum gamma R2 + sum beta R2 + sum gamma R1
  // and sum gamma R2 = sum gamma R1 + s sum gamma.  Q is taken from the end that is
  // nearer in the nearest image: beside the segment's line the other one cancels.
  // fast: far() holds and on_line() does not.
  __device__ __forceinline__ void gradient(double ux, double uy, double uz, double L, bool fast,
                                           bool skip_main, double *dR, double *dS) const {
    const double hx = sy * uz - sz * uy, hy = sz * ux - sx * uz, hz = sx * uy - sy * ux;
    double f0 = 0., g0 = 0.;
    double fX = 0., fY = 0., fZ = 0., aX = 0., aY = 0., aZ = 0.;  // sums of f R1, alpha R1,
    double bX = 0., bY = 0., bZ = 0., cX = 0., cY = 0., cZ = 0.;  // beta R2 and gamma R1
    if (fast) {
      const bool near2 = least<PX>(tx) + least<PY>(ty) + least<PZ>(tz) <
                         least<PX>(px) + least<PY>(py) + least<PZ>(pz);
#pragma unroll 1  // a third of the code and registers: three blocks per SM
      for (int a = 0; a < PX; a++) {
        const double sh = PX == 3 ? (a - 1) * L : 0., xa = rx[PX / 2] + sh, ea = ex[PX / 2] + sh,
                     pa = xa * xa, ga = xa * ea, ta = ea * ea, qa = (near2 ? ea : xa) * hx;
        double fa = 0., aa = 0., ba = 0., ca = 0.;  // sums over the shifts (b, k) of this a
#pragma unroll
        for (int b = 0; b < PY; b++) {
          // from r and e again, an fma where p, t and g need an addition: those
          // arrays would take more registers than there are
          const double pxy = fma(ry[b], ry[b], pa), gxy = fma(ry[b], ey[b], ga),
                       txy = fma(ey[b], ey[b], ta), qxy = fma(near2 ? ey[b] : ry[b], hy, qa);
          double fb = 0., ab = 0., bb = 0., cb = 0.;
#pragma unroll
          for (int k = 0; k < PZ; k++) {
            double A = fma(rz[k], rz[k], pxy), B = fma(ez[k], ez[k], txy);
            double d = fma(rz[k], ez[k], gxy), Q = fma(near2 ? ez[k] : rz[k], hz, qxy);
            const bool own = skip_main && (a * PY + b) * PZ + k == NI / 2;
            if (own) A = B = d = 1.;
            if (own) Q = 0.;
            SegD t = seg_d_pos(A, B, d, Q);
            if (own) t.f = 0.;
            fb += t.f; ab += t.fA2; bb += t.fB2; cb += t.fd;
            fZ = fma(t.f, rz[k], fZ);
            aZ = fma(t.fA2, rz[k], aZ);
            bZ = fma(t.fB2, ez[k], bZ);
            cZ = fma(t.fd, rz[k], cZ);
          }
          fa += fb; aa += ab; ba += bb; ca += cb;
          fY = fma(fb, ry[b], fY);
          aY = fma(ab, ry[b], aY);
          bY = fma(bb, ey[b], bY);
          cY = fma(cb, ry[b], cY);
        }
        f0 += fa; g0 += ca;
        fX = fma(fa, xa, fX);
        aX = fma(aa, xa, aX);
        bX = fma(ba, ea, bX);
        cX = fma(ca, xa, cX);
      }
    } else {
#pragma unroll 1
      for (int m = 0; m < NI; m++) {
        if (skip_main && m == NI / 2) continue;
        double R1[3], R2[3], cr[3], A, B, d;
        image(m, L, R1, R2);
        image_term(R1, R2, A, B, d, cr);
        const SegD t = seg_d_any(A, B, d, cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2],
                                 cr[0] * ux + cr[1] * uy + cr[2] * uz);
        const double al = t.fA2, be = t.fB2, ga = t.fd;
        f0 += t.f; g0 += ga;
        fX += t.f * R1[0]; fY += t.f * R1[1]; fZ += t.f * R1[2];
        aX += al * R1[0]; aY += al * R1[1]; aZ += al * R1[2];
        bX += be * R2[0]; bY += be * R2[1]; bZ += be * R2[2];
        cX += ga * R1[0]; cY += ga * R1[1]; cZ += ga * R1[2];
      }
    }
    dS[0] = bX + cX + (uy * fZ - uz * fY);
    dS[1] = bY + cY + (uz * fX - ux * fZ);
    dS[2] = bZ + cZ + (ux * fY - uy * fX);
    dR[0] = fma(hx, f0, fma(sx, g0, aX + cX)) + (bX + cX);
    dR[1] = fma(hy, f0, fma(sy, g0, aY + cY)) + (bY + cY);
    dR[2] = fma(hz, f0, fma(sz, g0, aZ + cZ)) + (bZ + cZ);
  }
};
