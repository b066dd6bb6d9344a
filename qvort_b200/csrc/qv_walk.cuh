// qv_walk.cuh -- device helpers shared by the Barnes-Hut walks (single system
// and batched forest): the reference's FP64 distance and opening test
// (src/tree.f90:350-365, 394), the compensated FP32 accumulator and the
// stack entry of the mixed-precision walk.
#pragma once
#include "qv_f32x2.cuh"
#include "qv_f64.cuh"
#include "qv_internal.cuh"

__device__ __forceinline__ double shift_of(int m, double L) {
  return m == 0 ? 0. : (m > 0 ? L : -L);
}

// The k-th image to walk: the images across a face first, then those across an
// edge, then a corner.  A face's image holds the near field of the groups beside
// that face, whose tasks are the longest of all the images'; taken in the
// reference's loop order the last of them started when most of the walk was done
// and set its end.  Only the order of independent tasks: every task keeps its
// slot, and the sums are added in the reference's order.
static __constant__ unsigned char QV_IMG_ORDER26[26] = {4,  10, 12, 13, 15, 21, 1,  3,  5,
                                                        7,  9,  11, 14, 16, 18, 20, 22, 24,
                                                        0,  2,  6,  8,  17, 19, 23, 25};
static __constant__ unsigned char QV_IMG_ORDER8[8] = {1, 3, 4, 6, 0, 2, 5, 7};
template <int BC>
__device__ __forceinline__ int image_at(int k) {
  return BC == QV_BC_PERIODIC ? QV_IMG_ORDER26[k] : BC == QV_BC_OPENX ? QV_IMG_ORDER8[k] : k;
}

// The order of the FP64 walks' tasks: the longest first.  Rows of one task per
// target group: row 0 the unshifted image's root child that holds the group (its
// near field), then the images across a face, the other root children, the
// other images.  The slot of the group that starts at target q in row `row`; r =
// the root's header.  Tangle, FP64 velocity: 0.759 -> 0.740 ms (the mixed walk's
// tasks in this order: no change).
template <int BC, int NS>
__device__ __forceinline__ int task_slot(int row, int q, const WNode64 &r, const WNode64 *w64) {
  constexpr int NF = BC == QV_BC_PERIODIC ? 6 : BC == QV_BC_OPENX ? 4 : BC == QV_BC_OPENXY ? 2 : 0;
  if (row >= 1 && row <= NF) return NS + image_at<BC>(row - 1);
  if (row >= NF + NS) return NS + image_at<BC>(row - NS);
  // targets lie in the order of the root's children
  int home = 0;
  for (int c = 0, end = 0; c < r.nchild; c++) {
    end += w64[r.child_first + c].count;
    if (q < end) {
      home = c;
      break;
    }
  }
  return row == 0 ? home : (home + row - NF) % NS;
}

// dist = |x_i - (cent + shift)| in the reference's operation order.
__device__ __forceinline__ double exact_dist(const double *xi, const WNode64 &h, const double *s) {
  double d0 = __dsub_rn(xi[0], __dadd_rn(h.cx, s[0]));
  double d1 = __dsub_rn(xi[1], __dadd_rn(h.cy, s[1]));
  double d2 = __dsub_rn(xi[2], __dadd_rn(h.cz, s[2]));
  return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(d0, d0), __dmul_rn(d1, d1)), __dmul_rn(d2, d2)));
}

// theta test of src/tree.f90:354-365,394 on a non-leaf node; true = open.
__device__ __forceinline__ bool exact_open(double dist, const WNode64 &h, double theta_tree,
                                           int extra) {
  double th;
  if (extra) {
    double r = __dsub_rn(dist, h.geo);
    th = r > 0. ? __ddiv_rn(h.width, r) : __ddiv_rn(h.width, dist);
  } else {
    th = __ddiv_rn(h.width, dist);
  }
  return !(th < theta_tree);
}

// The root's opening test while its header holds the centroid estimate of
// k_root_est, whose distance from the exact (sequentially summed) centroid is
// at most delta.  Moving the centroid by delta moves dist and geo by at most
// delta each, so the test is decided for every centroid in that ball when
// width/(dist - geo) stays on one side of tree_theta over dist - geo +- 2 delta
// (and width/dist over dist +- delta where dist <= geo is possible); the margin
// also carries a relative 1e-14 for the rounding of the test itself.  A decided
// test returns its answer.  An undecided one returns "open" (the lane walks the
// image) and sets `unc`; the fix-up after the walk takes the exact decision and
// drops the image's sum if the root was in fact far.  delta = 0: the header
// holds the exact centroid and this is the reference's test.
__device__ __forceinline__ bool root_open(const double *xi, const WNode64 &r, const double *s,
                                          double theta, int extra, double delta, bool &unc) {
  const double dist = exact_dist(xi, r, s);
  const bool open = exact_open(dist, r, theta, extra);
  if (!(delta > 0.)) return open;
  const double m = delta + 1e-14 * (dist + r.geo + r.width);
  bool cfar, copen;
  if (extra) {
    const double rl = dist - r.geo - 2. * m, rh = dist - r.geo + 2. * m;
    cfar = rl > 0. && r.width < theta * rl;
    copen = (rh <= 0. || r.width >= theta * rh) && (rl > 0. || r.width >= theta * (dist + m));
  } else {
    cfar = r.width < theta * (dist - m);
    copen = r.width >= theta * (dist + m);
  }
  if (cfar) return false;
  if (copen) return true;
  unc = true;
  return true;
}

__device__ __forceinline__ void cross3(const double *a, const double *b, double *c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

struct Kahan3w {
  float s[3], c[3];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < 3; k++) s[k] = c[k] = 0.f;
  }
  __device__ __forceinline__ void add(float a0, float a1, float a2) {
    float a[3] = {a0, a1, a2};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      float y = __fsub_rn(a[k], c[k]);
      float t = __fadd_rn(s[k], y);
      c[k] = __fsub_rn(__fsub_rn(t, s[k]), y);
      s[k] = t;
    }
  }
  __device__ __forceinline__ double get(int k) const { return (double)s[k] - (double)c[k]; }
};

// Kahan3w for two targets at once: (s, c) hold target a in .x and target b
// in .y.  add() applies the scalar update's operations to both halves and
// keeps the new values only where the half's flag is set, so each half goes
// through exactly the sequence of updates a Kahan3w of its own would.
struct Kahan3x2 {
  float2 s[3], c[3];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < 3; k++) s[k] = c[k] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void add(float2 a0, float2 a1, float2 a2, bool fx, bool fy) {
    const float2 a[3] = {a0, a1, a2};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float2 y = sub2(a[k], c[k]);
      const float2 t = add2(s[k], y);
      const float2 cn = sub2(sub2(t, s[k]), y);
      s[k].x = fx ? t.x : s[k].x;
      s[k].y = fy ? t.y : s[k].y;
      c[k].x = fx ? cn.x : c[k].x;
      c[k].y = fy ? cn.y : c[k].y;
    }
  }
  // half H alone (a leaf pair of one of the two targets)
  template <int H>
  __device__ __forceinline__ void add1(float a0, float a1, float a2) {
    const float a[3] = {a0, a1, a2};
#pragma unroll
    for (int k = 0; k < 3; k++) {
      float &sk = H ? s[k].y : s[k].x;
      float &ck = H ? c[k].y : c[k].x;
      const float y = __fsub_rn(a[k], ck);
      const float t = __fadd_rn(sk, y);
      ck = __fsub_rn(__fsub_rn(t, sk), y);
      sk = t;
    }
  }
  __device__ __forceinline__ double get(int h, int k) const {
    return (double)pick(s[k], h) - (double)pick(c[k], h);
  }
};

// One target of a lane's pair: its point index and links.
struct PairTarget {
  int i, bi, fi;  // point index (0-based), behind, infront; bi = fi = -1 if not live
};

// Far-field term of a cell (payload P, d2 = |v|^2) for the targets of a pair that
// accept it (fa, fb).
__device__ __forceinline__ void far_pair(const WPay32 &P, float2 v0, float2 v1, float2 v2, float2 d2,
                                         bool fa, bool fb, Kahan3x2 &k0) {
  // below 1e-25 the powers overflow either way
  const float2 rd = make_float2(rsqrt_normal(d2.x), rsqrt_normal(d2.y));
  const float2 rd2 = mul2(rd, rd), rd3 = mul2(rd2, rd), rd5 = mul2(rd3, rd2);
  const float2 z0 = fma2(v0, bc2(P.C[0]), fma2(v1, bc2(P.C[3]), mul2(v2, bc2(P.C[6]))));
  const float2 z1 = fma2(v0, bc2(P.C[1]), fma2(v1, bc2(P.C[4]), mul2(v2, bc2(P.C[7]))));
  const float2 z2 = fma2(v0, bc2(P.C[2]), fma2(v1, bc2(P.C[5]), mul2(v2, bc2(P.C[8]))));
  const float2 cx = sub2(fma2(bc2(P.a[1]), v2, mul2(bc2(-P.a[2]), v1)), bc2(P.b[0]));
  const float2 cy = sub2(fma2(bc2(P.a[2]), v0, mul2(bc2(-P.a[0]), v2)), bc2(P.b[1]));
  const float2 cz = sub2(fma2(bc2(P.a[0]), v1, mul2(bc2(-P.a[1]), v0)), bc2(P.b[2]));
  const float2 wx = fma2(v1, z2, mul2(neg2(v2), z1));
  const float2 wy = fma2(v2, z0, mul2(neg2(v0), z2));
  const float2 wz = fma2(v0, z1, mul2(neg2(v1), z0));
  const float2 t5 = mul2(bc2(3.f), rd5);
  k0.add(fma2(cx, rd3, mul2(wx, t5)), fma2(cy, rd3, mul2(wy, t5)),
         fma2(cz, rd3, mul2(wz, t5)), fa, fb);
}

// Stack entry: the child's FP32 header, fetched when the child is pushed so
// that popping it costs a shared-memory read instead of a dependent global load,
// and the lane masks of the targets that opened the parent (mask: the warp's
// first 32 targets; mask2: the second 32 where a lane carries two).
struct __align__(16) StkEnt {
  WNode32 h;
  int node;
  unsigned mask, mask2;
  int pad;
};


// ------------------------------------------------------------ FP64 walks
// Stack entry of the FP64 walks: the child's centroid shifted to the task's
// image and the squared opening radius, made by the lane that pushes it, so
// that a pop reads shared memory and the distance vector -- x_i - (cent + shift),
// rounded as the reference's -- serves both the opening test and the far term.
struct __align__(16) StkEnt64 {
  double cx, cy, cz;
  // squared distance above rhi: the node is taken whole; below rlo: opened; in
  // between (and where no radius is valid: rhi = inf, rlo = -1) the reference's
  // expression decides
  double rhi, rlo;
  int node;
  unsigned mask;
  int child_first, nc;  // nc: children, or -1 for a one-point leaf
  int jb, pad;
};

// Opening test theta = width / (dist - geo) < tree_theta (geo = 0 without the
// extra correction) as dist^2 > rc2, rc = geo + width / tree_theta.  A cell's
// centroid lies inside it, so geo <= (sqrt 3 / 2) width, and a distance below
// geo gives width / dist >= 2 / sqrt 3: for tree_theta < 1.15 the two agree.
// The relative margin of 1e-11 on either side is far above the rounding of
// both (dist - geo loses at most a factor two); the reference's rounded
// expression decides inside it, so every decision is the reference's.
__device__ __forceinline__ void fill_ent64(StkEnt64 &E, const WNode64 &h, int node, unsigned mask,
                                           const double *s, double inv_theta, bool extra,
                                           bool sure) {
  E.cx = h.cx + s[0]; E.cy = h.cy + s[1]; E.cz = h.cz + s[2];
  const double rc = (extra ? h.geo : 0.) + h.width * inv_theta, rc2 = rc * rc;
  E.rhi = sure ? rc2 * (1. + 1e-11) : __longlong_as_double(0x7ff0000000000000ll);
  E.rlo = sure ? rc2 * (1. - 1e-11) : -1.;
  E.node = node;
  E.mask = mask;
  E.child_first = h.child_first;
  E.nc = h.count == 1 ? -1 : h.nchild;
  E.jb = h.jb;
}

// Far cell (src/tree.f90:397-411): (circ x v - w) / d^3 + 3 v x (C^T v) / d^5,
// v = x - (cent + shift), d2 = |v|^2 > 0, added to acc.
__device__ __forceinline__ void far_term64(double v0, double v1, double v2, double d2,
                                           const WPay64 &P, double *acc) {
  const double r = rsqrt_pos(d2), r2 = r * r, r3 = r2 * r, t5 = 3. * r3 * r2;
  const double z0 = fma(v0, P.C[0], fma(v1, P.C[3], v2 * P.C[6]));
  const double z1 = fma(v0, P.C[1], fma(v1, P.C[4], v2 * P.C[7]));
  const double z2 = fma(v0, P.C[2], fma(v1, P.C[5], v2 * P.C[8]));
  const double cx = fma(P.a[1], v2, fma(-P.a[2], v1, -P.b[0]));
  const double cy = fma(P.a[2], v0, fma(-P.a[0], v2, -P.b[1]));
  const double cz = fma(P.a[0], v1, fma(-P.a[1], v0, -P.b[2]));
  acc[0] = fma(cx, r3, fma(fma(v1, z2, -v2 * z1), t5, acc[0]));
  acc[1] = fma(cy, r3, fma(fma(v2, z0, -v0 * z2), t5, acc[1]));
  acc[2] = fma(cz, r3, fma(fma(v0, z1, -v1 * z0), t5, acc[2]));
}

// One-point leaf (src/tree.f90:380-390): the straight segment from R1 to R2 =
// R1 + s, scale times its term added to acc, where the target lies off the
// segment (R1.R2 well above 0): the form there neither cancels nor divides by
// a small number.  false: beside or on the segment, nothing added -- the caller
// takes the reference's expression.
__device__ __forceinline__ bool leaf_term64(double r1x, double r1y, double r1z, double r2x,
                                            double r2y, double r2z, double sx, double sy, double sz,
                                            double scale, double *acc) {
  const double d = r1x * r2x + r1y * r2y + r1z * r2z;
  if (!(d > 0.0625 * (sx * sx + sy * sy + sz * sz))) return false;
  const double A = r1x * r1x + r1y * r1y + r1z * r1z, B = r2x * r2x + r2y * r2y + r2z * r2z;
  const double f = seg_f_pos(A, B, d) * scale;
  acc[0] = fma(f, r1y * sz - r1z * sy, acc[0]);
  acc[1] = fma(f, r1z * sx - r1x * sz, acc[1]);
  acc[2] = fma(f, r1x * sy - r1y * sx, acc[2]);
  return true;
}
