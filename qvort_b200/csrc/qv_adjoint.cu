// qv_adjoint.cu -- hand-written derivatives of the velocity path.
//
// qv_velocity_vjp: x_bar = J^T u_bar for u = calc_velocity(x) (src/timestep.f90:
// 180-309) through every piece of it:
//   * the local LIA term (forward-mode dual numbers over its 9- or 15-value
//     ghost stencil, the same templated formula as the velocity),
//   * the direct sum (hand-derived gradients of the straight-segment term, one
//     pass over the pairs for both ends, no atomics),
//   * or the Barnes-Hut walk with the topology of the last build frozen
//     (hand-derived leaf and monopole+dipole gradients; the gradients that
//     belong to a source cell are reduced over the warp and added to a per-node
//     adjoint of (cent, circ, Cij), which a last kernel distributes to the
//     cell's points through the moment definitions of src/tree.f90:146-179),
//   * and the ghost gather (ghosti_i = x_infront(i) etc., src/periodic.f90:23-31),
//     whose adjoint is a gather over behind/infront.
// qv_energy_grad: energy_info (src/diagnostic.f90:259-280) and its gradients
// with respect to x and u.
// qv_field_velocity: biot_savart_general(_shift) (src/timestep.f90:516-563) at
// arbitrary points and its exact gradient, in place of the central
// differences of velocity_quasip (src/hamiltonian.f90:65-89).
//
// Segment term (leaf form of src/tree.f90:380-390, the same function as the
// direct form of src/timestep.f90:472-479):
//   u = f R1 x R2,  f = (a+b)/P,  P = a b (a b + d),  a=|R1|, b=|R2|, d=R1.R2
// For an upstream g:  Q = g.(R1 x R2),
//   dQ/dR1 = R2 x g,  dQ/dR2 = g x R1,
//   df/da = (P - (a+b) b(2ab+d))/P^2,  df/db = (P - (a+b) a(2ab+d))/P^2,
//   df/dd = -(a+b) ab / P^2,
//   grad_R1 (f Q) = Q (df/da R1/a + df/dd R2) + f (R2 x g),
//   grad_R2 (f Q) = Q (df/db R2/b + df/dd R1) + f (g x R1).
// Far cell (monopole + dipole, restated as in the walk):
//   u = r3 (circ x v - w) + 3 r5 v x z,  z = C^T v,  r3 = |v|^-3, r5 = |v|^-5,
//   grad_v (g.u) = -3 r5 (g.a) v + r3 g x circ - 15 r7 (g.b) v + 3 r5 (z x g + C (g x v)),
//   with a = circ x v - w, b = v x z;  d/dcirc = r3 v x g;  d/dw = -r3 g;
//   d/dz = 3 r5 g x v  ->  d/dC(p,l) = v_p (d/dz)_l.
#include <algorithm>
#include <vector>

#include "qv_internal.cuh"
#include "qv_ab.cuh"
#include "qv_f64.cuh"
#include "qv_lia.cuh"
#include "qv_walk.cuh"

static inline int nblk(long n, int t) { return (int)((n + t - 1) / t); }

// ------------------------------------------------------------- segment term
__device__ __forceinline__ void seg_grad(const double *R1, const double *R2, const double *g,
                                         double *gR1, double *gR2) {
  double a = sqrt(R1[0] * R1[0] + R1[1] * R1[1] + R1[2] * R1[2]);
  double b = sqrt(R2[0] * R2[0] + R2[1] * R2[1] + R2[2] * R2[2]);
  double d = R1[0] * R2[0] + R1[1] * R2[1] + R1[2] * R2[2];
  double ab = a * b;
  double P = ab * (ab + d);
  double f = (a + b) / P;
  double cr[3] = {R1[1] * R2[2] - R1[2] * R2[1], R1[2] * R2[0] - R1[0] * R2[2],
                  R1[0] * R2[1] - R1[1] * R2[0]};
  double Q = g[0] * cr[0] + g[1] * cr[1] + g[2] * cr[2];
  double P2 = P * P, t = 2. * ab + d;
  double dfa = (P - (a + b) * b * t) / P2, dfb = (P - (a + b) * a * t) / P2;
  double dfd = -(a + b) * ab / P2;
  double r2g[3] = {R2[1] * g[2] - R2[2] * g[1], R2[2] * g[0] - R2[0] * g[2],
                   R2[0] * g[1] - R2[1] * g[0]};
  double gr1[3] = {g[1] * R1[2] - g[2] * R1[1], g[2] * R1[0] - g[0] * R1[2],
                   g[0] * R1[1] - g[1] * R1[0]};
#pragma unroll
  for (int c = 0; c < 3; c++) {
    gR1[c] = Q * (dfa * R1[c] / a + dfd * R2[c]) + f * r2g[c];
    gR2[c] = Q * (dfb * R2[c] / b + dfd * R1[c]) + f * gr1[c];
  }
}

// ------------------------------------------------------------------- LIA
// Seeds input component k (0..14: x, gi, gb, gii, gbb) and returns the
// directional derivative of the local velocity.
__device__ void lia_vjp_point(int vel, int order, int fixed, double G, double a, const double *X,
                              const double *GI, const double *GB, const double *GII,
                              const double *GBB, const double *ub, double *bar) {
  const int nin = order == 4 ? 15 : 9;
  for (int k = 0; k < 15; k++) bar[k] = 0.;
  for (int k = 0; k < nin; k++) {
    Dual in[15];
    const double *src[5] = {X, GI, GB, GII, GBB};
    for (int q = 0; q < 15; q++) in[q] = Dual(src[q / 3][q % 3], q == k ? 1. : 0.);
    Dual out[3];
    lia_term(vel, order, fixed, G, a, in, in + 3, in + 6, in + 9, in + 12, out);
    bar[k] = ub[0] * out[0].d + ub[1] * out[1].d + ub[2] * out[2].d;
  }
}

__global__ void k_lia_vjp(int n, const double *__restrict__ x, const int *__restrict__ inf,
                          const double *__restrict__ gi, const double *__restrict__ gb,
                          const double *__restrict__ gii, const double *__restrict__ gbb,
                          const double *__restrict__ ubar, int vel, int order, int fixed, double G,
                          double a, double *xb, double *gib, double *gbb_, double *giib,
                          double *gbbb) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double bar[15];
  if (inf[i] == 0) {
    for (int k = 0; k < 15; k++) bar[k] = 0.;
  } else {
    double X[3], GI[3], GB[3], GII[3], GBB[3], ub[3];
    for (int c = 0; c < 3; c++) {
      X[c] = x[3 * i + c]; GI[c] = gi[3 * i + c]; GB[c] = gb[3 * i + c];
      GII[c] = gii[3 * i + c]; GBB[c] = gbb[3 * i + c]; ub[c] = ubar[3 * i + c];
    }
    lia_vjp_point(vel, order, fixed, G, a, X, GI, GB, GII, GBB, ub, bar);
  }
  for (int c = 0; c < 3; c++) {
    xb[3 * i + c] = bar[c];
    gib[3 * i + c] = bar[3 + c];
    gbb_[3 * i + c] = bar[6 + c];
    giib[3 * i + c] = bar[9 + c];
    gbbb[3 * i + c] = bar[12 + c];
  }
}

// ------------------------------------------------------------ direct sum
// One pass over all (source, target) pairs gives both ends' gradients: a thread
// holds one source and sums its own (dL/dx_j at fixed s, dL/ds) over a chunk of
// targets, while each target's gradient -- minus the sum over sources -- is
// reduced over the warp (12 shuffles a target against 27 images x ~50 FP64
// operations a lane) and over the block's warps in shared memory.  Partial
// sums per (source block, target) and per (target chunk, source) are added in
// a fixed order by k_dvjp_reduce, so results are deterministic, with no
// atomics.  A two-pass split (a thread per target, then a thread per source)
// evaluates every pair twice.  Bound: FP64 issue.  6,400 points, 27 images:
// velocity and gradient together took 333 ms with two passes, divisions in every
// image term and 50 blocks; 6.9 ms now, 2 of them the velocity (this kernel 4.7,
// 77 % of the FP64 rate at 52 operations a pair and image; the x shifts unrolled
// took 255 registers, two blocks per SM and 0.4 ms more).
#define VT 128  // sources per block
#define VG 32   // targets per shared-memory tile
size_t g_dvjp_part = QV_DVJP_PART;  // qv_test_direct_split lowers it

// Sum of (v0, v1, v2) over the warp: lanes 0, 8 and 16 return the three sums.
__device__ __forceinline__ double warp_sum3(double v0, double v1, double v2, int lane) {
  const bool hi = lane & 16, md = lane & 8;
  double a = hi ? v2 : v0, b = hi ? 0. : v1;
  a += __shfl_xor_sync(0xffffffffu, hi ? v0 : v2, 16);
  b += __shfl_xor_sync(0xffffffffu, hi ? v1 : 0., 16);
  double r = md ? b : a;
  r += __shfl_xor_sync(0xffffffffu, md ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  return r;
}

// Targets t_lo..t_hi (positions in act); tpart: (source blocks) x (t_hi - t_lo)
// x 3, spart: (target chunks) x na x 6.
template <int BC>
__global__ void __launch_bounds__(VT, 3) k_dvjp(int na, const int *__restrict__ act,
                                                const double *__restrict__ x,
                                                const double *__restrict__ gi,
                                                const int *__restrict__ beh,
                                                const double *__restrict__ ubar, double gfac,
                                                double L, int t_lo, int t_hi, int chunk_len,
                                                double *tpart, double *spart) {
  __shared__ double tx[VG][3], tg[VG][3], red[VT / 32][VG][3];
  __shared__ int tb[VG], ti[VG];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int q = blockIdx.x * VT + threadIdx.x;
  const bool live = q < na;
  const int j = live ? act[q] : 0, jj = j + 1;
  double xj[3] = {0., 0., 0.}, gj[3] = {0., 0., 0.}, s[3], dx[3] = {0., 0., 0.}, dg[3] = {0., 0., 0.};
  if (live)
#pragma unroll
    for (int c = 0; c < 3; c++) { xj[c] = x[3 * j + c]; gj[c] = gi[3 * j + c]; }
#pragma unroll
  for (int c = 0; c < 3; c++) s[c] = gj[c] - xj[c];
  const double c2 = s[0] * s[0] + s[1] * s[1] + s[2] * s[2];
  const int t0 = t_lo + blockIdx.y * chunk_len, t1 = min(t_hi, t0 + chunk_len);
  for (int t = t0; t < t1; t += VG) {
    const int m = min(VG, t1 - t);
    __syncthreads();  // the last tile's sums are out
    for (int e = threadIdx.x; e < 3 * m; e += VT) {
      const int k = e / 3, c = e - 3 * k, i = act[t + k];
      tx[k][c] = x[3 * i + c];
      tg[k][c] = gfac * ubar[3 * i + c];
      if (c == 0) {
        tb[k] = beh[i];
        ti[k] = i + 1;
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < m; k++) {
      const Seg64<BC> e(xj[0] - tx[k][0], xj[1] - tx[k][1], xj[2] - tx[k][2], gj[0] - tx[k][0],
                        gj[1] - tx[k][1], gj[2] - tx[k][2], s[0], s[1], s[2], c2, L);
      // src/timestep.f90:471, 496
      const bool own = jj == ti[k], skip = !live || jj == tb[k] || (own && e.NI == 1);
      const bool fast = __all_sync(0xffffffffu, skip || (e.far(own, L) && !e.on_line()));
      double dR[3] = {0., 0., 0.}, dS[3];
      if (!skip) {
        e.gradient(tg[k][0], tg[k][1], tg[k][2], L, fast, own, dR, dS);
#pragma unroll
        for (int c = 0; c < 3; c++) { dx[c] += dR[c] - dS[c]; dg[c] += dS[c]; }
      }
      __syncwarp();
      const double r = warp_sum3(dR[0], dR[1], dR[2], lane);
      if ((lane & 7) == 0 && lane < 24) red[wid][k][lane >> 3] = r;
    }
    __syncthreads();
    double *o = tpart + ((size_t)blockIdx.x * (t_hi - t_lo) + (t - t_lo)) * 3;
    for (int e = threadIdx.x; e < 3 * m; e += VT) {
      double v = 0.;
#pragma unroll
      for (int w = 0; w < VT / 32; w++) v += red[w][e / 3][e % 3];
      o[e] = v;
    }
  }
  if (live) {
    double *o = spart + ((size_t)blockIdx.y * na + q) * 6;
#pragma unroll
    for (int c = 0; c < 3; c++) { o[c] = dx[c]; o[3 + c] = dg[c]; }
  }
}

// Adds a slab's partial sums to the point adjoints: one thread per component.
__global__ void k_dvjp_reduce(int na, const int *__restrict__ act, int t_lo, int t_hi, int nsb,
                              int nchunk, const double *__restrict__ tpart,
                              const double *__restrict__ spart, double *xb, double *gib) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * na) return;
  const int q = e / 3, c = e - 3 * q, o = 3 * act[q] + c;
  double sx = 0., sg = 0., st = 0.;
#pragma unroll 8
  for (int k = 0; k < nchunk; k++) {
    const double *p = spart + ((size_t)k * na + q) * 6 + c;
    sx += p[0];
    sg += p[3];
  }
  if (q >= t_lo && q < t_hi) {
    const size_t stride = 3 * (size_t)(t_hi - t_lo);
    const double *p = tpart + (e - 3 * t_lo);
#pragma unroll 8
    for (int k = 0; k < nsb; k++) st += p[k * stride];
  }
  xb[o] += sx - st;
  gib[o] += sg;
}

// ------------------------------------------------------------ tree walk
// The velocity walk again, with the opened cells held: one node at a time for 32
// targets.  A node's adjoint (cent, circ, C: 15 values) is the sum over its
// targets: a halving butterfly (16 exchanges where summing each value on its
// own took 75) leaves the sums spread over the lanes, which add them to the
// node's record (128 bytes) with one atomic instruction.  The opening test and
// the far-field gradient need one reciprocal square root, as in the velocity
// walk.
//
// Bound: instruction issue (a third of it FP64).  50,000 points, 27 images, theta
// 0.4: 2.28 ms with a rounded square root and division per test, 15 separate
// warp sums and 15 atomics by one lane per node; 0.97 ms now.  Two or four
// nodes at a time for 16 or 8 targets send two to four times the atomics,
// which then meet on the top nodes' L2 lines (1.2 and 3.5 ms; 1.0 and 1.15 with
// 16 copies of those nodes' records).
#define AW 4
#define ANSPLIT 8
#define NBS 16  // doubles per node adjoint record: cent 3, circ 3, C 9, unused

struct WalkVjpArgs {
  int n_act, ngroups, stk_cap;
  const int *perm, *inf, *beh;
  const double *x, *ubar;
  const WNode64 *w64;
  const WPay64 *p64;
  double L, theta, gfac;
  int extra;
  double *xb, *gib, *nb;  // nb: per-node adjoints (NBS doubles each)
};

// Sums the NV values of v (16 or 8) over the warp by halving: v[0] of lane l
// becomes the sum of value l / (32 / NV).
template <int NV>
__device__ __forceinline__ void warp_sums(double *v, int lane) {
  int n = NV;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool up = lane & o;
#pragma unroll
      for (int k = 0; k < NV / 2; k++) {
        if (k >= n) break;
        const double keep = up ? v[k + n] : v[k], send = up ? v[k] : v[k + n];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
}

// Gradients of g . f (R1 x R2) for a straight segment s = R2 - R1 off the target (d =
// R1.R2 > 0): dR with respect to both ends together, dS to the second alone (see
// Seg64::gradient).
__device__ __forceinline__ void seg_gradient_pos(const double *R1, const double *R2,
                                                 const double *s, const double *g, double A,
                                                 double B, double d, double *dR, double *dS) {
  const double h[3] = {s[1] * g[2] - s[2] * g[1], s[2] * g[0] - s[0] * g[2],
                       s[0] * g[1] - s[1] * g[0]};
  const double gr[3] = {g[1] * R1[2] - g[2] * R1[1], g[2] * R1[0] - g[0] * R1[2],
                        g[0] * R1[1] - g[1] * R1[0]};
  const double Q = (B < A ? R2[0] : R1[0]) * h[0] + (B < A ? R2[1] : R1[1]) * h[1] +
                   (B < A ? R2[2] : R1[2]) * h[2];
  const SegD t = seg_d_pos(A, B, d, Q);
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const double v = fma(t.fB2, R2[c], t.fd * R1[c]);
    dS[c] = fma(t.f, gr[c], v);
    dR[c] = fma(t.f, h[c], fma(t.fA2, R1[c], t.fd * R2[c])) + v;
  }
}

template <int BC>
__global__ void __launch_bounds__(AW * 32, 4) k_walk_vjp(WalkVjpArgs a) {
  constexpr int NIMG = BC == QV_BC_PERIODIC ? 26 : BC == QV_BC_OPENX ? 8 : BC == QV_BC_OPENXY ? 2 : 0;
  extern __shared__ int2 stk_adj[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int2 *st = stk_adj + wid * a.stk_cap;
  const double ith = 1. / a.theta;
  const bool sure = !a.extra || a.theta < 1.15;
  const int items = a.ngroups * (ANSPLIT + NIMG);
  for (int item = blockIdx.x * AW + wid; item < items; item += gridDim.x * AW) {
    const WNode64 r = a.w64[0];
    const int row = item / a.ngroups, q0 = (item - row * a.ngroups) * 32, q = q0 + lane;
    const int sl = task_slot<BC, ANSPLIT>(row, q0, r, a.w64);
    const bool live = q < a.n_act;
    const int i = live ? a.perm[q] : 0;
    double xi[3] = {0., 0., 0.}, gu[3] = {0., 0., 0.}, acc[3] = {0., 0., 0.};
    int bi = -1, fi = -1, ii = -1;
    if (live) {
#pragma unroll
      for (int c = 0; c < 3; c++) { xi[c] = a.x[3 * i + c]; gu[c] = a.gfac * a.ubar[3 * i + c]; }
      bi = a.beh[i]; fi = a.inf[i]; ii = i + 1;
    }
    int ma = 0, mb = 0, mc = 0;
    if (sl >= ANSPLIT) qv_img_shift(BC, sl - ANSPLIT, &ma, &mb, &mc);
    const double s[3] = {shift_of(ma, a.L), shift_of(mb, a.L), shift_of(mc, a.L)};
    // the root's own decision; the unshifted image's tasks then take one child
    const bool lone = r.count == 1;
    const bool go = live && (lone ? sl == 0 || sl >= ANSPLIT
                                  : exact_open(exact_dist(xi, r, s), r, a.theta, a.extra));
    const unsigned rm = __ballot_sync(0xffffffffu, go);
    const int c0 = lone ? 0 : r.child_first + (sl < ANSPLIT ? sl : 0);
    const int c1 = lone ? 1 : r.child_first + (sl < ANSPLIT ? min(r.nchild, sl + 1) : r.nchild);
    int top = rm ? max(0, c1 - c0) : 0;
    if (lane < top) st[lane] = make_int2(c0 + lane, (int)rm);
    __syncwarp();
    while (top > 0) {
      top--;
      const int2 e = st[top];
      __syncwarp();
      const int node = e.x;
      const bool in = (((unsigned)e.y) >> lane) & 1u;
      const WNode64 h = a.w64[node];
      // x - (cent + shift) with the velocity walk's roundings: x - shift - cent
      // differs by a unit of the box, which for a small cell is more than the
      // margin of the test below
      const double v[3] = {xi[0] - (h.cx + s[0]), xi[1] - (h.cy + s[1]), xi[2] - (h.cz + s[2])};
      const double d2 = fma(v[0], v[0], fma(v[1], v[1], v[2] * v[2]));
      bool open = false, far = false, leaf = false;
      double w[16];
      const WPay64 &P = a.p64[node];
      if (in && h.count == 1) {
        const int j = h.jb;
        leaf = j != ii && j != bi && j != fi;
      } else if (in) {
        const double rc = fma(h.width, ith, a.extra ? h.geo : 0.), rc2 = rc * rc;
        // as in the velocity walk (fill_ent64): the reference's expression near rc
        open = !sure || !(fabs(d2 - rc2) > 1e-11 * rc2)
                   ? exact_open(exact_dist(xi, h, s), h, a.theta, a.extra)
                   : d2 < rc2;
        far = !open && node != 0;
      }
      if (__any_sync(0xffffffffu, leaf)) {
#pragma unroll
        for (int k = 0; k < 8; k++) w[k] = 0.;
        if (leaf) {
          double dR[3], dS[3];
          const double R[3] = {-v[0], -v[1], -v[2]};
          double sv[3], R2[3];
#pragma unroll
          for (int c = 0; c < 3; c++) sv[c] = P.b[c] - P.a[c];
#pragma unroll
          for (int c = 0; c < 3; c++) R2[c] = P.b[c] + s[c] - xi[c];
          const double d = R[0] * R2[0] + R[1] * R2[1] + R[2] * R2[2];
          if (d > 0.0625 * (sv[0] * sv[0] + sv[1] * sv[1] + sv[2] * sv[2])) {
            seg_gradient_pos(R, R2, sv, gu, d2, R2[0] * R2[0] + R2[1] * R2[1] + R2[2] * R2[2], d,
                             dR, dS);
          } else {  // beside the segment
            double g1[3], E1[3], E2[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
              E1[c] = P.a[c] + s[c] - xi[c];
              E2[c] = P.b[c] + s[c] - xi[c];
            }
            seg_grad(E1, E2, gu, g1, dS);
#pragma unroll
            for (int c = 0; c < 3; c++) dR[c] = g1[c] + dS[c];
          }
#pragma unroll
          for (int c = 0; c < 3; c++) {
            acc[c] -= dR[c];
            w[c] = dR[c] - dS[c];
            w[3 + c] = dS[c];
          }
        }
        warp_sums<8>(w, lane);
        const int m = lane >> 2;  // the value this lane holds
        if ((lane & 3) == 0 && m < 6) atomicAdd(&(m < 3 ? a.xb : a.gib)[3 * h.first + m % 3], w[0]);
        continue;
      }
      if (__any_sync(0xffffffffu, far)) {
#pragma unroll
        for (int k = 0; k < 16; k++) w[k] = 0.;
        if (far) {
          const double r1 = rsqrt_pos(d2), r2 = r1 * r1, r3 = r2 * r1, r5 = r3 * r2;
          const double p5 = 3. * r5;
          double z[3], av[3], bv[3];
#pragma unroll
          for (int l = 0; l < 3; l++) z[l] = fma(v[0], P.C[l], fma(v[1], P.C[3 + l], v[2] * P.C[6 + l]));
          av[0] = fma(P.a[1], v[2], fma(-P.a[2], v[1], -P.b[0]));
          av[1] = fma(P.a[2], v[0], fma(-P.a[0], v[2], -P.b[1]));
          av[2] = fma(P.a[0], v[1], fma(-P.a[1], v[0], -P.b[2]));
          cross3(v, z, bv);
          const double ga = gu[0] * av[0] + gu[1] * av[1] + gu[2] * av[2];
          const double gb = gu[0] * bv[0] + gu[1] * bv[1] + gu[2] * bv[2];
          double gxc[3], zxg[3], gxv[3];
          cross3(gu, P.a, gxc);
          cross3(z, gu, zxg);
          cross3(gu, v, gxv);
          const double kv = -p5 * fma(5. * r2, gb, ga);
#pragma unroll
          for (int c = 0; c < 3; c++) {
            const double Cg = fma(P.C[3 * c], gxv[0], fma(P.C[3 * c + 1], gxv[1], P.C[3 * c + 2] * gxv[2]));
            const double gv = fma(kv, v[c], fma(r3, gxc[c], p5 * (zxg[c] + Cg)));
            acc[c] += gv;
            w[c] = -gv;               // cent
            w[3 + c] = -r3 * gxv[c];  // circ: r3 v x g
          }
          // C(p, l): v_p (3 r5 g x v)_l, and w_0 = C12 - C21, w_1 = C20 - C02,
          // w_2 = C01 - C10 with adjoint -r3 g
          const double zb[3] = {p5 * gxv[0], p5 * gxv[1], p5 * gxv[2]};
          const double wb[3] = {-r3 * gu[0], -r3 * gu[1], -r3 * gu[2]};
          w[6] = v[0] * zb[0];
          w[7] = fma(v[0], zb[1], wb[2]);
          w[8] = fma(v[0], zb[2], -wb[1]);
          w[9] = fma(v[1], zb[0], -wb[2]);
          w[10] = v[1] * zb[1];
          w[11] = fma(v[1], zb[2], wb[0]);
          w[12] = fma(v[2], zb[0], wb[1]);
          w[13] = fma(v[2], zb[1], -wb[0]);
          w[14] = v[2] * zb[2];
        }
        warp_sums<16>(w, lane);
        if (!(lane & 1) && lane < 30) atomicAdd(a.nb + NBS * (size_t)node + (lane >> 1), w[0]);
      }
      const unsigned om = __ballot_sync(0xffffffffu, open);
      if (om) {
        int nc = h.nchild;
        if (top + nc > a.stk_cap) nc = 0;  // unreachable: the cap follows the tree depth
        if (lane < nc) st[top + lane] = make_int2(h.child_first + nc - 1 - lane, (int)om);
        top += nc;
        __syncwarp();
      }
    }
    if (live)
#pragma unroll
      for (int c = 0; c < 3; c++) atomicAdd(&a.xb[3 * i + c], acc[c]);
  }
}

// Node adjoint -> point adjoints through cent = sum x / n, circ = sum (gi - x),
// C = sum x (gi - x)^T - cent circ^T (src/tree.f90:154-179): the points t0, t0 +
// step, ... of node k.
struct MomentArgs {
  const int *level, *start, *count, *ord;
  int cap_pts;
  const double *x, *gi, *cent, *circ, *nb;
  double *xb, *gib;
};
__device__ __forceinline__ void moment_vjp(const MomentArgs &a, int k, int t0, int step) {
  const int n = a.count[k];
  if (n == 1) return;  // a leaf's gradients went to its point
  const double *B = a.nb + NBS * (size_t)k;
  double Cb[9], cb[3], qb[3];
  bool any = false;
  for (int t = 0; t < 15; t++) any |= B[t] != 0.;
  if (!any) return;
  for (int t = 0; t < 9; t++) Cb[t] = B[6 + t];
  const double *cent = a.cent + 3 * (size_t)k, *circ = a.circ + 3 * (size_t)k;
  // C = C_raw - cent circ^T
  for (int r = 0; r < 3; r++) {
    cb[r] = B[r] - (Cb[3 * r] * circ[0] + Cb[3 * r + 1] * circ[1] + Cb[3 * r + 2] * circ[2]);
    qb[r] = B[3 + r] - (Cb[r] * cent[0] + Cb[3 + r] * cent[1] + Cb[6 + r] * cent[2]);
  }
  for (int c = 0; c < 3; c++) cb[c] /= n;
  const int *o = a.ord + (size_t)a.level[k] * a.cap_pts + a.start[k];
  for (int t = t0; t < n; t += step) {
    const int p = o[t];
    double X[3], s[3];
    for (int c = 0; c < 3; c++) { X[c] = a.x[3 * p + c]; s[c] = a.gi[3 * p + c] - X[c]; }
    for (int c = 0; c < 3; c++) {
      const double Cs = Cb[3 * c] * s[0] + Cb[3 * c + 1] * s[1] + Cb[3 * c + 2] * s[2];  // (C_b s)_c
      const double CtX = Cb[c] * X[0] + Cb[3 + c] * X[1] + Cb[6 + c] * X[2];          // (C_b^T x)_c
      atomicAdd(&a.xb[3 * p + c], cb[c] - qb[c] + Cs - CtX);
      atomicAdd(&a.gib[3 * p + c], qb[c] + CtX);
    }
  }
}
// Nodes k0 .. n_nodes - 1, eight to a block: a warp each, and the block's warps
// together where a node holds more than MV_BIG points.
#define MV_BIG 128
__global__ void __launch_bounds__(256) k_moment_vjp(MomentArgs a, int k0, int n_nodes) {
  const int b0 = k0 + blockIdx.x * 8, k = b0 + (threadIdx.x >> 5);
  if (k < n_nodes && a.count[k] <= MV_BIG) moment_vjp(a, k, threadIdx.x & 31, 32);
  for (int e = b0; e < min(b0 + 8, n_nodes); e++)
    if (a.count[e] > MV_BIG) moment_vjp(a, e, threadIdx.x, 256);
}
// The nodes of the first levels (1 .. n - 1) hold most of the points each: MV_SPLIT
// blocks per node.  A warp for a root child of 6,000 points was a chain of 200
// gathers and atomics, 285 us at 50,000 points; 28 us for these and 89 for the
// others now.
#define MV_TOP 585  // levels 0 to 3 of a full octree
#define MV_SPLIT 16
__global__ void __launch_bounds__(256) k_moment_vjp_top(MomentArgs a, int n) {
  const int k = 1 + blockIdx.x;
  if (k < n) moment_vjp(a, k, blockIdx.y * 256 + threadIdx.x, 256 * MV_SPLIT);
}

// Ghost adjoint: gi_i = x_infront(i), gb_i = x_behind(i), gii_i = x_infront(infront(i)),
// gbb_i = x_behind(behind(i)) (shifts by +-L are constants).
__global__ void k_ghost_vjp(int n, const int *__restrict__ inf, const int *__restrict__ beh,
                            const double *__restrict__ xb, const double *__restrict__ gib,
                            const double *__restrict__ gbb_, const double *__restrict__ giib,
                            const double *__restrict__ gbbb, double *out) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  if (inf[p] == 0) {
    for (int c = 0; c < 3; c++) out[3 * p + c] = 0.;
    return;
  }
  int b = beh[p] - 1, f = inf[p] - 1, bb = beh[b] - 1, ff = inf[f] - 1;
  for (int c = 0; c < 3; c++)
    out[3 * p + c] = xb[3 * p + c] + gib[3 * b + c] + gbb_[3 * f + c] + giib[3 * bb + c] + gbbb[3 * ff + c];
}

// ------------------------------------------------------------------ energy
// W_q = u_q . (x_q x s'_q), l_q = |x_q - ghosti_q|.
template <typename T>
__device__ __forceinline__ T energy_w(int order, const T *X, const T *GI, const T *GB,
                                      const T *GII, const T *GBB, const double *u) {
  T s1[3], s2[3];
  lia_derivs(order, X, GI, GB, GII, GBB, s1, s2);
  T c0 = X[1] * s1[2] - X[2] * s1[1], c1 = X[2] * s1[0] - X[0] * s1[2], c2 = X[0] * s1[1] - X[1] * s1[0];
  return u[0] * c0 + u[1] * c1 + u[2] * c2;
}

__global__ void k_energy_w(int n, const double *__restrict__ x, const double *__restrict__ u,
                           const int *__restrict__ inf, const double *__restrict__ gi,
                           const double *__restrict__ gb, const double *__restrict__ gii,
                           const double *__restrict__ gbb, int order, double *W, double *ell) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n || inf[q] == 0) return;
  double X[3], GI[3], GB[3], GII[3], GBB[3], U[3];
  for (int c = 0; c < 3; c++) {
    X[c] = x[3 * q + c]; GI[c] = gi[3 * q + c]; GB[c] = gb[3 * q + c];
    GII[c] = gii[3 * q + c]; GBB[c] = gbb[3 * q + c]; U[c] = u[3 * q + c];
  }
  W[q] = energy_w(order, X, GI, GB, GII, GBB, U);
  ell[q] = lia_dist(X, GI);
}

// E = G sum_i 0.5 l_i (W_i + W_infront(i)); per point the term, the u
// gradient G 0.5 (l_q + l_behind(q)) x_q x s'_q, and the stencil gradients.
__global__ void k_energy_grad(int n, const double *__restrict__ x, const double *__restrict__ u,
                              const int *__restrict__ inf, const int *__restrict__ beh,
                              const double *__restrict__ gi, const double *__restrict__ gb,
                              const double *__restrict__ gii, const double *__restrict__ gbb,
                              const double *__restrict__ W, const double *__restrict__ ell,
                              int order, double G, double *eterm, double *ub, double *xb,
                              double *gib, double *gbb_, double *giib, double *gbbb) {
  int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  for (int c = 0; c < 3; c++) {
    ub[3 * q + c] = 0.; xb[3 * q + c] = 0.; gib[3 * q + c] = 0.; gbb_[3 * q + c] = 0.;
    giib[3 * q + c] = 0.; gbbb[3 * q + c] = 0.;
  }
  eterm[q] = 0.;
  if (inf[q] == 0) return;
  int a = inf[q] - 1, b = beh[q] - 1;
  double X[3], GI[3], GB[3], GII[3], GBB[3], U[3];
  for (int c = 0; c < 3; c++) {
    X[c] = x[3 * q + c]; GI[c] = gi[3 * q + c]; GB[c] = gb[3 * q + c];
    GII[c] = gii[3 * q + c]; GBB[c] = gbb[3 * q + c]; U[c] = u[3 * q + c];
  }
  eterm[q] = 0.5 * ell[q] * (W[q] + W[a]);
  double cW = G * 0.5 * (ell[q] + ell[b]);
  double cL = G * 0.5 * (W[q] + W[a]);
  // dE/du_q = cW (x_q x s'_q)
  double s1[3], s2[3];
  lia_derivs(order, X, GI, GB, GII, GBB, s1, s2);
  ub[3 * q] = cW * (X[1] * s1[2] - X[2] * s1[1]);
  ub[3 * q + 1] = cW * (X[2] * s1[0] - X[0] * s1[2]);
  ub[3 * q + 2] = cW * (X[0] * s1[1] - X[1] * s1[0]);
  // dE/d(stencil) through W_q
  const int nin = order == 4 ? 15 : 9;
  double bar[15];
  for (int k = 0; k < 15; k++) bar[k] = 0.;
  for (int k = 0; k < nin; k++) {
    Dual in[15];
    const double *src[5] = {X, GI, GB, GII, GBB};
    for (int t = 0; t < 15; t++) in[t] = Dual(src[t / 3][t % 3], t == k ? 1. : 0.);
    bar[k] = cW * energy_w(order, in, in + 3, in + 6, in + 9, in + 12, U).d;
  }
  // dE/dl_q: l_q = |x_q - gi_q|
  for (int c = 0; c < 3; c++) {
    double dl = ell[q] > 0. ? (X[c] - GI[c]) / ell[q] : 0.;
    bar[c] += cL * dl;
    bar[3 + c] -= cL * dl;
  }
  for (int c = 0; c < 3; c++) {
    xb[3 * q + c] = bar[c]; gib[3 * q + c] = bar[3 + c]; gbb_[3 * q + c] = bar[6 + c];
    giib[3 * q + c] = bar[9 + c]; gbbb[3 * q + c] = bar[12 + c];
  }
}

// ------------------------------------------------------------- field points
// biot_savart_general(_shift) at m points (src/timestep.f90:516-563): every
// active segment, no skip; and the exact gradient du_i/dx_k of the unshifted
// sum (what velocity_quasip differentiates) or (GI) of the full periodic sum.
//
// A warp takes one point and one chunk of the sources, a lane per source: a
// handful of points (quasiparticles) then still fills the chip, where a thread
// per point left 100 threads with 23,500 sources x 27 images each.  The FW
// warps of a block take neighbouring points and the same chunk, which they
// meet in L1.  Bound: FP64 issue.  100 points, 23,500 sources, 27 images: 302
// ms with a thread per point, 0.23 ms per call now (copies included).
#define FW 4
#define FV 12  // values per point: u (3), du/dx row-major (9)
#define QV_FIELD_SLAB (1 << 20)  // points per launch (bounds the partial sums: 101 MB)

// du_r/dx_k -= d(f c_r)/dR_k for one term, c = R1 x s and both ends moving together:
// with v = (2 fA + fd) R1 + (2 fB + fd) R2, d(f c_r)/dR_k = c_r v_k + f eps(r,k,l) s_l.
__device__ __forceinline__ void add_jacobian(const SegD &t, const double *R1, const double *R2,
                                             double sx, double sy, double sz, const double *c,
                                             double *J) {
  const double p = t.fA2 + t.fd, q = t.fB2 + t.fd;
  const double vx = fma(p, R1[0], q * R2[0]), vy = fma(p, R1[1], q * R2[1]),
               vz = fma(p, R1[2], q * R2[2]);
  J[0] -= c[0] * vx;
  J[1] -= fma(c[0], vy, t.f * sz);
  J[2] -= fma(c[0], vz, -t.f * sy);
  J[3] -= fma(c[1], vx, -t.f * sz);
  J[4] -= c[1] * vy;
  J[5] -= fma(c[1], vz, t.f * sx);
  J[6] -= fma(c[2], vx, t.f * sy);
  J[7] -= fma(c[2], vy, -t.f * sx);
  J[8] -= c[2] * vz;
}

template <int BC, bool GI>
__global__ void __launch_bounds__(FW * 32) k_field(int m, const double *__restrict__ pts, int na,
                                                   const double *__restrict__ src, int chunk_len,
                                                   int nchunk, double L, double *part) {
  const int lane = threadIdx.x & 31;
  const int g = blockIdx.x / nchunk, chunk = blockIdx.x - g * nchunk;
  const int t = g * FW + (threadIdx.x >> 5);
  if (t >= m) return;  // whole warps
  const double X = pts[3 * (size_t)t], Y = pts[3 * (size_t)t + 1], Z = pts[3 * (size_t)t + 2];
  double v[FV];
#pragma unroll
  for (int k = 0; k < FV; k++) v[k] = 0.;
  const int j0 = chunk * chunk_len, j1 = min(na, j0 + chunk_len);
#pragma unroll 1
  for (int j = j0 + lane; j - lane < j1; j += 32) {
    const bool live = j < j1;
    const double2 *s = reinterpret_cast<const double2 *>(src + 8 * (size_t)(live ? j : j0));
    const double2 s0 = s[0], s1 = s[1], s2 = s[2];
    const double sx = s1.y, sy = s2.x, sz = s2.y, c = s[3].x;
    const double dx = s0.x - X, dy = s0.y - Y, dz = s1.x - Z;
    const Seg64<BC> e(dx, dy, dz, dx + sx, dy + sy, dz + sz, sx, sy, sz, c, L);
    const bool fast = __all_sync(0xffffffffu, !live || e.far(false, L));
    if (!live) continue;
    constexpr int NI = Seg64<BC>::NI;
    if (!GI) e.velocity(L, fast, false, v[0], v[1], v[2]);
#pragma unroll 1
    for (int im = GI ? 0 : NI / 2; im < (GI ? NI : NI / 2 + 1); im++) {
      double R1[3], R2[3], cr[3], A, B, d;
      e.image(im, L, R1, R2);
      e.image_term(R1, R2, A, B, d, cr);
      const double c2 = cr[0] * cr[0] + cr[1] * cr[1] + cr[2] * cr[2];
      // a point on the segment's line: no term (4ac - b^2 = 0, src/timestep.f90:531)
      if (c2 == 0.) continue;
      const SegD q = fast ? seg_d_pos(A, B, d, 1.) : seg_d_any(A, B, d, c2, 1.);
      if (GI) {
        v[0] += q.f * cr[0];
        v[1] += q.f * cr[1];
        v[2] += q.f * cr[2];
      }
      add_jacobian(q, R1, R2, sx, sy, sz, cr, v + 3);
    }
  }
#pragma unroll
  for (int k = 0; k < FV; k++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  }
  double *o = part + ((size_t)chunk * m + t) * FV;
#pragma unroll
  for (int k = 0; k < FV; k++)
    if (lane == k) o[k] = v[k];
}

// Sum of the chunks' partial values, a warp per value (lanes stride over the
// chunks, in a fixed order).
__global__ void k_field_reduce(int m, int nchunk, const double *__restrict__ part, double scale,
                               double *u, double *dudx) {
  const long e = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const long tot = (long)m * FV;
  if (e >= tot) return;
  double s = 0.;
  for (int k = lane; k < nchunk; k += 32) s += part[k * tot + e];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const long t = e / FV;
  const int k = (int)(e - t * FV);
  if (lane == 0) (k < 3 ? u[3 * t + k] : dudx[9 * t + (k - 3)]) = s * scale;
}

// ------------------------------------------------------------------ host side
static int adj_reserve(qv_ctx *c) {
  size_t v = sizeof(double) * 3 * (size_t)std::max(c->n, 1);
  if (c->adj_n >= c->n && c->adj_xb) return QV_OK;
  int rc;
  double **bufs[] = {&c->adj_xb, &c->adj_gib, &c->adj_gbb, &c->adj_giib, &c->adj_gbbb};
  for (double **b : bufs)
    if ((rc = qv_grow(c, (void **)b, v))) return rc;
  c->adj_n = c->n;
  return QV_OK;
}

// ------------------------------------------------------ Adams-Bashforth step
// The position update of pmotion (src/timestep.f90:48-71) followed by the wrap
// of enforce_periodic (src/periodic.f90:188-214), from device arrays, and its
// adjoint.  The forward takes the update kernel's operations (qv_ab.cuh), so a
// differentiable trajectory is bitwise the trajectory qv_step would make from
// the same velocities.  The rung is chosen by exact-zero tests of the history,
// piecewise constant in every input, and the wrap moves a point by a constant:
// the adjoint is x_bar = x_out_bar and (u, u1, u2, u3)_bar = the rung's
// coefficients times x_out_bar.  Empty slots (infront = 0) do not move.
__global__ void k_ab_fwd(int n, double dt, const double *__restrict__ x,
                         const double *__restrict__ u, const double *__restrict__ u1,
                         const double *__restrict__ u2, const double *__restrict__ u3,
                         const int *__restrict__ inf, int lo_axis, double L, double *xo) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (inf[i] == 0) {
    for (int c = 0; c < 3; c++) xo[3 * i + c] = x[3 * i + c];
    return;
  }
  double U1[3], U2[3], U3[3];
  for (int c = 0; c < 3; c++) {
    U1[c] = u1[3 * i + c]; U2[c] = u2[3 * i + c]; U3[c] = u3[3 * i + c];
  }
  const int rung = ab_rung(U1, U2, U3);
  for (int c = 0; c < 3; c++) {
    const double r = ab_update(rung, dt, x[3 * i + c], u[3 * i + c], U1[c], U2[c], U3[c]);
    xo[3 * i + c] = c >= lo_axis ? wrap_coord(r, L) : r;
  }
}

__global__ void k_ab_vjp(int n, double dt, const double *__restrict__ u1,
                         const double *__restrict__ u2, const double *__restrict__ u3,
                         const int *__restrict__ inf, const double *__restrict__ xob, double *xb,
                         double *ub, double *u1b, double *u2b, double *u3b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double k[4] = {0., 0., 0., 0.};
  if (inf[i] != 0) {
    double U1[3], U2[3], U3[3];
    for (int c = 0; c < 3; c++) {
      U1[c] = u1[3 * i + c]; U2[c] = u2[3 * i + c]; U3[c] = u3[3 * i + c];
    }
    ab_coef(ab_rung(U1, U2, U3), dt, k);
  }
  for (int c = 0; c < 3; c++) {
    const double g = xob[3 * i + c];
    xb[3 * i + c] = g;
    ub[3 * i + c] = k[0] * g;
    u1b[3 * i + c] = k[1] * g;
    u2b[3 * i + c] = k[2] * g;
    u3b[3 * i + c] = k[3] * g;
  }
}

static int ab_lo_axis(int bc) {
  return bc == QV_BC_PERIODIC ? 0 : bc == QV_BC_OPENX ? 1 : bc == QV_BC_OPENXY ? 2 : 3;
}

extern "C" int qv_ab_step_device(qv_ctx *c, int n, const double *x, const double *u,
                                 const double *u1, const double *u2, const double *u3,
                                 double *x_out) {
  if (!c) return QV_ERR_ARG;
  if (n != c->n) return qv_fail(c, QV_ERR_STATE, "qv_ab_step_device: %d slots, context holds %d", n, c->n);
  if (n == 0) return QV_OK;
  if (!x || !u || !u1 || !u2 || !u3 || !x_out) return qv_fail(c, QV_ERR_ARG, "null array");
  k_ab_fwd<<<nblk(n, 256), 256, 0, c->stream>>>(n, c->p.dt, x, u, u1, u2, u3, c->infront,
                                                ab_lo_axis(c->p.boundary), c->p.box_size, x_out);
  QV_LAUNCH_CHECK(c);
  QV_COUNT(c, 1);
  return QV_OK;
}

extern "C" int qv_ab_vjp_device(qv_ctx *c, int n, const double *u1, const double *u2,
                                const double *u3, const double *xbar_out, double *xbar,
                                double *ubar, double *u1bar, double *u2bar, double *u3bar) {
  if (!c) return QV_ERR_ARG;
  if (n != c->n) return qv_fail(c, QV_ERR_STATE, "qv_ab_vjp_device: %d slots, context holds %d", n, c->n);
  if (n == 0) return QV_OK;
  if (!u1 || !u2 || !u3 || !xbar_out || !xbar || !ubar || !u1bar || !u2bar || !u3bar)
    return qv_fail(c, QV_ERR_ARG, "null array");
  k_ab_vjp<<<nblk(n, 256), 256, 0, c->stream>>>(n, c->p.dt, u1, u2, u3, c->infront, xbar_out,
                                                xbar, ubar, u1bar, u2bar, u3bar);
  QV_LAUNCH_CHECK(c);
  QV_COUNT(c, 1);
  return QV_OK;
}

extern "C" int qv_velocity_vjp(qv_ctx *c, const double *ubar, double *xbar) {
  if (!c || !ubar || !xbar) return QV_ERR_ARG;
  if (c->n == 0) return QV_OK;
  int rc;
  if (!c->ghosts_valid)
    if ((rc = qv_launch_ghosts(c))) return rc;
  if ((rc = adj_reserve(c))) return rc;
  const qv_params &p = c->p;
  k_lia_vjp<<<nblk(c->n, 128), 128, 0, c->stream>>>(
      c->n, c->x, c->infront, c->gi, c->gb, c->gii, c->gbb, ubar, p.velocity, p.deriv_order,
      p.fixed_lia_beta, p.quant_circ, p.corea, c->adj_xb, c->adj_gib, c->adj_gbb, c->adj_giib,
      c->adj_gbbb);
  QV_LAUNCH_CHECK(c);
  QV_COUNT(c, 1);
  double gfac = p.quant_circ / (4. * QV_PI);
  if (p.velocity == QV_VEL_BS) {
    if ((rc = qv_compact_active(c))) return rc;
    int na = c->n_act;
    if (na > 0) {
      // Slabs of targets bound the partial sums: source blocks x targets x 24
      // bytes is 2 GB at 100,000 points, so above QV_DVJP_PART bytes the
      // targets are taken in several launches.
      const int nsb = nblk(na, VT);
      const size_t row = sizeof(double) * 3 * (size_t)nsb;
      const int slab = (int)std::min<size_t>(na, std::max<size_t>(VG, g_dvjp_part / row / VG * VG));
      // ten blocks per resident slot (3 per SM; with five the last wave cost 5 %),
      // each with enough pairs (targets x images) to outweigh its start and its
      // partial sums
      const int want = nblk(30L * c->sm_count, nsb);
      const int least = p.boundary == QV_BC_PERIODIC ? 8 : p.boundary == QV_BC_OPENX ? 16 : VG;
      const int chunk_len = nblk(nblk(slab, want), least) * least, nchunk = nblk(slab, chunk_len);
      const size_t tbytes = row * slab, sbytes = sizeof(double) * 6 * (size_t)na * nchunk;
      if (tbytes + sbytes > c->dpart_bytes) {
        c->dpart_bytes = 0;  // the old buffer goes first
        if ((rc = qv_grow(c, (void **)&c->dpart, tbytes + sbytes))) return rc;
        c->dpart_bytes = tbytes + sbytes;
      }
      double *tpart = c->dpart, *spart = c->dpart + tbytes / sizeof(double);
      for (int t_lo = 0; t_lo < na; t_lo += slab) {
        const int t_hi = std::min(na, t_lo + slab), nch = nblk(t_hi - t_lo, chunk_len);
        const dim3 grid(nsb, nch);
        switch (p.boundary) {
#define QV_DVJP(BCV)                                                                              \
  case BCV:                                                                                       \
    k_dvjp<BCV><<<grid, VT, 0, c->stream>>>(na, c->act, c->x, c->gi, c->behind, ubar, gfac,       \
                                            p.box_size, t_lo, t_hi, chunk_len, tpart, spart);     \
    break;
          QV_DVJP(QV_BC_OPEN)
          QV_DVJP(QV_BC_PERIODIC)
          QV_DVJP(QV_BC_OPENX)
          QV_DVJP(QV_BC_OPENXY)
#undef QV_DVJP
          default:
            return qv_fail(c, QV_ERR_UNSUPPORTED, "boundary %d", p.boundary);
        }
        QV_LAUNCH_CHECK(c);
        k_dvjp_reduce<<<nblk(3L * na, 128), 128, 0, c->stream>>>(
            na, c->act, t_lo, t_hi, nsb, nch, tpart, spart, c->adj_xb, c->adj_gib);
        QV_LAUNCH_CHECK(c);
        QV_COUNT(c, 2);
      }
    }
  } else if (p.velocity == QV_VEL_TREE) {
    if (!c->tree.valid)
      if ((rc = qv_launch_tree_build(c))) return rc;
    if ((rc = qv_tree_finalize_root(c))) return rc;
    TreeBuf &t = c->tree;
    size_t nbytes = sizeof(double) * NBS * (size_t)t.n_nodes;
    if (nbytes > c->adj_nb_bytes) {
      if ((rc = qv_grow(c, (void **)&c->adj_nb, nbytes))) return rc;
      c->adj_nb_bytes = nbytes;
    }
    QV_CUDA(c, cudaMemsetAsync(c->adj_nb, 0, nbytes, c->stream));
    if (t.n_act > 0) {
      WalkVjpArgs a;
      a.n_act = t.n_act; a.ngroups = (t.n_act + 31) / 32; a.perm = t.perm;
      a.inf = c->infront; a.beh = c->behind; a.x = c->x; a.ubar = ubar; a.w64 = t.w64; a.p64 = t.p64;
      a.L = p.box_size; a.theta = p.tree_theta; a.gfac = gfac; a.extra = p.tree_extra_correction;
      a.xb = c->adj_xb; a.gib = c->adj_gib; a.nb = c->adj_nb;
      a.stk_cap = 7 * (t.depth + 1) + 8;  // as in the velocity walk
      const size_t smem = sizeof(int2) * a.stk_cap * AW;
      int nimg = qv_img_count(p.boundary);
      long items = (long)a.ngroups * (ANSPLIT + nimg);
      int nb = (int)std::min<long>((items + AW - 1) / AW, 64L * c->sm_count);
      const void *f = nullptr;
      switch (p.boundary) {
        case QV_BC_OPEN: f = (const void *)k_walk_vjp<QV_BC_OPEN>; break;
        case QV_BC_PERIODIC: f = (const void *)k_walk_vjp<QV_BC_PERIODIC>; break;
        case QV_BC_OPENX: f = (const void *)k_walk_vjp<QV_BC_OPENX>; break;
        case QV_BC_OPENXY: f = (const void *)k_walk_vjp<QV_BC_OPENXY>; break;
        default: return qv_fail(c, QV_ERR_UNSUPPORTED, "boundary %d", p.boundary);
      }
      if (smem > 48 * 1024)
        if ((rc = qv_smem_optin(c, f))) return rc;
      void *args[] = {&a};
      QV_CUDA(c, cudaLaunchKernel(f, dim3(nb), dim3(AW * 32), args, smem, c->stream));
      QV_LAUNCH_CHECK(c);
      if (t.n_nodes > 1) {
        MomentArgs m;
        m.level = t.level; m.start = t.start; m.count = t.count; m.ord = t.ord;
        m.cap_pts = t.cap_pts; m.x = c->x; m.gi = c->gi; m.cent = t.cent; m.circ = t.circ;
        m.nb = c->adj_nb; m.xb = c->adj_xb; m.gib = c->adj_gib;
        const int ntop = std::min(t.n_nodes, MV_TOP);
        k_moment_vjp_top<<<dim3(ntop - 1, MV_SPLIT), 256, 0, c->stream>>>(m, ntop);
        QV_COUNT(c, 1);
        if (t.n_nodes > ntop) {
          k_moment_vjp<<<nblk(t.n_nodes - ntop, 8), 256, 0, c->stream>>>(m, ntop, t.n_nodes);
          QV_COUNT(c, 1);
        }
        QV_LAUNCH_CHECK(c);
      }
      QV_COUNT(c, 1);
    }
  }
  k_ghost_vjp<<<nblk(c->n, 256), 256, 0, c->stream>>>(c->n, c->infront, c->behind, c->adj_xb,
                                                      c->adj_gib, c->adj_gbb, c->adj_giib,
                                                      c->adj_gbbb, xbar);
  QV_LAUNCH_CHECK(c);
  QV_COUNT(c, 1);
  QV_CUDA(c, cudaStreamSynchronize(c->stream));
  return QV_OK;
}

extern "C" int qv_energy_grad(qv_ctx *c, const double *u, double *energy, double *xbar,
                              double *ubar) {
  if (!c || !u || !energy || !xbar || !ubar) return QV_ERR_ARG;
  if (c->n == 0) { *energy = 0.; return QV_OK; }
  int rc;
  if (!c->ghosts_valid)
    if ((rc = qv_launch_ghosts(c))) return rc;
  if ((rc = adj_reserve(c))) return rc;
  int n = c->n;
  double *W = nullptr;
  QV_CUDA(c, cudaMalloc((void **)&W, sizeof(double) * 3 * (size_t)n));
  double *ell = W + n, *eterm = W + 2 * (size_t)n;
  QV_CUDA(c, cudaMemsetAsync(W, 0, sizeof(double) * 3 * (size_t)n, c->stream));
  k_energy_w<<<nblk(n, 128), 128, 0, c->stream>>>(n, c->x, u, c->infront, c->gi, c->gb, c->gii,
                                                  c->gbb, c->p.deriv_order, W, ell);
  k_energy_grad<<<nblk(n, 128), 128, 0, c->stream>>>(
      n, c->x, u, c->infront, c->behind, c->gi, c->gb, c->gii, c->gbb, W, ell, c->p.deriv_order,
      c->p.quant_circ, eterm, ubar, c->adj_xb, c->adj_gib, c->adj_gbb, c->adj_giib, c->adj_gbbb);
  k_ghost_vjp<<<nblk(n, 256), 256, 0, c->stream>>>(n, c->infront, c->behind, c->adj_xb,
                                                   c->adj_gib, c->adj_gbb, c->adj_giib,
                                                   c->adj_gbbb, xbar);
  QV_LAUNCH_CHECK(c);
  QV_COUNT(c, 3);
  std::vector<double> h(n);
  QV_CUDA(c, cudaMemcpyAsync(h.data(), eterm, sizeof(double) * n, cudaMemcpyDeviceToHost, c->stream));
  QV_CUDA(c, cudaStreamSynchronize(c->stream));
  QV_CUDA(c, cudaFree(W));
  // Neumaier-compensated sum of the per-point terms: the energy of a loss is
  // differenced across nearby states, and a plain sequential sum's rounding
  // (up to n u sum|t|) would dominate a difference quotient at small steps;
  // qv_energy keeps the reference's sequential order
  double e = 0., comp = 0.;
  for (int i = 0; i < n; i++) {
    const double t = e + h[i];
    comp += fabs(e) >= fabs(h[i]) ? (e - t) + h[i] : (h[i] - t) + e;
    e = t;
  }
  *energy = (e + comp) * c->p.quant_circ;
  return QV_OK;
}

int qv_pack_sources64(qv_ctx *c);

extern "C" int qv_field_velocity(qv_ctx *c, int m, const double *pts, int grad_images, double *u,
                                 double *dudx) {
  if (!c || m < 0 || (m > 0 && (!pts || !u || !dudx))) return QV_ERR_ARG;
  if (m == 0) return QV_OK;
  int rc;
  if (!c->ghosts_valid)
    if ((rc = qv_launch_ghosts(c))) return rc;
  if ((rc = qv_compact_active(c))) return rc;
  if ((rc = qv_pack_sources64(c))) return rc;
  const int na = c->n_act;
  // about four warps for each of the chip's FP64-saturating slots (16 per SM);
  // a chunk holds at least one source per lane
  const int slab = std::min(m, QV_FIELD_SLAB);
  const int want = (int)std::max(1L, 64L * c->sm_count / slab);
  const int chunk_len = std::max(1, nblk(nblk(na, want), 32)) * 32;
  const int nchunk = std::max(1, nblk(na, chunk_len));
  const size_t np = 3 * (size_t)m;
  // points, results and a slab's partial sums
  FieldBuf buf(c);
  if ((rc = buf.reserve(sizeof(double) * (5 * np + FV * (size_t)slab * nchunk)))) return rc;
  double *dp = c->field_buf, *du = dp + np, *dj = du + np, *part = dj + 3 * np;
  QV_CUDA(c, cudaMemcpyAsync(dp, pts, sizeof(double) * np, cudaMemcpyHostToDevice, c->stream));
  const double L = c->p.box_size;
  for (int lo = 0; lo < m; lo += slab) {
    const int ms = std::min(slab, m - lo);
    const double *p = dp + 3 * (size_t)lo;
    const unsigned nb = (unsigned)nblk(ms, FW) * nchunk;
    switch (c->p.boundary) {
#define QV_FIELD_CASE(BCV)                                                                        \
  case BCV:                                                                                       \
    if (grad_images && BCV != QV_BC_OPEN)                                                         \
      k_field<BCV, true><<<nb, FW * 32, 0, c->stream>>>(ms, p, na, c->src64, chunk_len, nchunk, L, \
                                                        part);                                    \
    else                                                                                          \
      k_field<BCV, false><<<nb, FW * 32, 0, c->stream>>>(ms, p, na, c->src64, chunk_len, nchunk,  \
                                                         L, part);                                \
    break;
      QV_FIELD_CASE(QV_BC_OPEN)
      QV_FIELD_CASE(QV_BC_PERIODIC)
      QV_FIELD_CASE(QV_BC_OPENX)
      QV_FIELD_CASE(QV_BC_OPENXY)
#undef QV_FIELD_CASE
      default: return qv_fail(c, QV_ERR_UNSUPPORTED, "boundary %d", c->p.boundary);
    }
    QV_LAUNCH_CHECK(c);
    k_field_reduce<<<(unsigned)(((size_t)ms * FV * 32 + 255) / 256), 256, 0, c->stream>>>(
        ms, nchunk, part, c->p.quant_circ / (4. * QV_PI), du + 3 * (size_t)lo, dj + 9 * (size_t)lo);
    QV_LAUNCH_CHECK(c);
    QV_COUNT(c, 2);
  }
  QV_CUDA(c, cudaMemcpyAsync(u, du, sizeof(double) * np, cudaMemcpyDeviceToHost, c->stream));
  QV_CUDA(c, cudaMemcpyAsync(dudx, dj, sizeof(double) * 9 * (size_t)m, cudaMemcpyDeviceToHost,
                             c->stream));
  QV_CUDA(c, cudaStreamSynchronize(c->stream));
  return QV_OK;
}
