// cn.cu -- K-CN: Crank-Nicolson steps.
//
// Replaces CrankNicholson::solveStep (src/crancNicholson.cpp:17-105) with the
// default ParaxialEquation (F = G = H = 1, J = 0, src/paraxialEquation.cpp:
// 3-21) and ThomasAlgorithm::solve (include/thomasAlgorithm.tpp:2-32).  A CTA
// (or a cluster) owns one problem; the field stays on chip for every step of
// the launch.  Three kernels:
//   cn_const_kernel   z-invariant media, Dirichlet ends;
//   cn_planes_kernel  media sampled per step, Dirichlet ends, a window of steps
//                     factored ahead by cn_pivot_kernel and cn_table_kernel;
//   cn_kernel         everything else (transparent ends, media sampled for few
//                     steps), step by step:
//   1. each thread builds the matrix rows of its chunk of M consecutive points
//      (diag, rhs; sub-diagonal constant) with the reference's operation
//      order, rounded op by op, so the coefficients equal the reference's;
//   2. each thread eliminates its chunk interior in registers (a partition
//      method: interior x_i = y_i + p_i x_first + q_i x_last) and writes the
//      two boundary equations of its chunk into a reduced system of 2T
//      unknowns;
//   3. the CTA solves the reduced system by cyclic reduction in shared memory;
//   4. each thread reconstructs its interior.
// The solves run in FP64 in both storage precisions: with rho = dz/(k dx^2)
// of a few hundred the system is only weakly diagonally dominant.  They differ
// from the reference's serial Thomas sweep in rounding; the step matrix is
// well conditioned (Cayley transform, condition ~ rho), so the difference
// stays near machine precision.
#include "pxp_complex.cuh"
#include "flux.cuh"
#include "pxp_kernels.h"
#include <algorithm>
#include <cstdlib>
#include <cooperative_groups.h>

#include "tridiag.cuh"

namespace cg = cooperative_groups;

namespace pxp {

// Diagonal of row i and its right-hand side (exact FP64, reference operation
// order).
__device__ __forceinline__ double2 cn_diag(double delta, double beta, double rho, double r) {
  // fval*1.0 + 0.25*(H+ + H-)*g*i*rho + 0.5*(beta*r + i*delta*r)
  double im_a = __dmul_rn(0.5, rho);              // 0.25*(1+1)*1 = 0.5, *i, *rho
  double br = __dmul_rn(beta, r);
  double dr = __dmul_rn(delta, r);
  double2 t = mk(__dmul_rn(0.5, br), __dmul_rn(0.5, dr));
  return mk(__dadd_rn(1.0, t.x), __dadd_rn(im_a, t.y));
}

__device__ __forceinline__ double2 cn_rhs(double2 left, double2 center, double2 right,
                                          double deltaPrev, double betaPrev, double rho,
                                          double r) {
  // rhs = left*H-'*g' + right*H+'*g'; rhs *= 0.25*i*rho
  double2 s = cx_add_rn(left, right);
  double q = __dmul_rn(0.25, rho);
  double2 rhs = cx_mul_rn(s, mk(0.0, q));
  // rhs -= 0.25*center*i*rho*(H+' + H-')*g
  double2 c4 = cx_scale_rn(center, 0.25);
  double2 t = cx_mul_rn(c4, mk(0.0, 1.0));
  t = cx_scale_rn(t, rho);
  t = cx_scale_rn(t, 2.0);
  rhs = cx_sub_rn(rhs, t);
  // rhs += (1.0*f' - 0.5*(beta'*r + i*delta'*r)) * center
  double2 h = mk(__dmul_rn(0.5, __dmul_rn(betaPrev, r)), __dmul_rn(0.5, __dmul_rn(deltaPrev, r)));
  // libstdc++ evaluates (double - complex) as (-y) + x
  double2 coef = mk(__dadd_rn(-h.x, 1.0), -h.y);
  return cx_add_rn(rhs, cx_mul_rn(coef, center));
}

// Transparent boundary (CrankNicholson::applyTBCOneSide,
// src/crancNicholson.cpp:136-148) with H- = g = 1.
__device__ __forceinline__ void cn_tbc(double2 outer, double2 inner, double rho, double2 &diag,
                                       double2 &rhs) {
  double2 ratio = cx_div_rn(outer, inner);
  double lr = log(hypot(ratio.x, ratio.y));
  double ar = atan2(ratio.y, ratio.x);
  double2 kdx = cx_div_rn(mk(lr, ar), mk(0.0, 1.0));
  if (kdx.x < 0.0) kdx.x = 0.0;
  double2 ik = cx_mul_rn(mk(0.0, 1.0), kdx);
  double e = exp(ik.x);
  double sn, cs;
  sincos(ik.y, &sn, &cs);
  double2 ex = mk(e * cs, e * sn);
  double2 coef = cx_mul_rn(mk(0.0, __dmul_rn(0.25, rho)), ex);
  diag = cx_sub_rn(diag, coef);
  rhs = cx_add_rn(rhs, cx_mul_rn(coef, outer));
}

template <typename R, int M, int T, bool FLUX>
__global__ void __launch_bounds__(T) cn_kernel(const CnJob *__restrict__ jobs, int step0_ov,
                                              int nsteps_ov) {
  using C = typename Cx<R>::T;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double flux_red[2][flux_slots<T>()];
  CnJob job = jobs[blockIdx.x];
  if (nsteps_ov >= 0) {
    job.step0 = step0_ov;
    job.nsteps = nsteps_ov;
  }
  const int n = job.n;  // == M * T
  // rows at and beyond nreal pad the system to M * T: diagonal kCnPad, zero
  // right-hand side and zero field, so they decouple from row nreal - 1 to
  // within |sub|^2 / kCnPad (the field beyond the grid is the Dirichlet zero)
  const int nreal = job.n_real > 0 ? job.n_real : n;
  const int nr = 2 * T;
  double2 *ra = reinterpret_cast<double2 *>(smem_raw);
  double2 *rb = ra + nr;
  double2 *rc = rb + nr;
  double2 *rd = rc + nr;
  C *u = reinterpret_cast<C *>(rd + nr);
  const int t = threadIdx.x;
  C *field = reinterpret_cast<C *>(job.field);
  for (int i = t; i < n; i += T) u[i] = i < nreal ? field[i] : C{};
  __syncthreads();
  const double rho = job.rho, r = job.r;
  const double2 sub = mk(-0.0, __dmul_rn(-0.25, rho));  // -0.25*i*rho*H-*g
  C *saves = reinterpret_cast<C *>(job.saves);
  const int s0 = t * M;

  for (int st = 0; st < job.nsteps; ++st) {
    const int step = job.step0 + st;
    // this step's flux window, loaded early so its latency hides behind the step
    int2 fw;
    const bool flux = FLUX && flux_window(job.flux, step, fw);
    const long long moff = job.mat_stride * (long long)(step - job.mat_step0);
    // ---- 1. rows of this chunk
    double2 dg[M], rh[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
      int i = s0 + m;
      if (i >= nreal) {
        dg[m] = mk(kCnPad, 0.0);
        rh[m] = mk(0.0, 0.0);
        continue;
      }
      double2 center = to_d(u[i]);
      double2 left = i > 0 ? to_d(u[i - 1]) : mk(0.0, 0.0);
      double2 right = i < nreal - 1 ? to_d(u[i + 1]) : mk(0.0, 0.0);
      double de = job.delta[moff + i], be = job.beta[moff + i];
      double dp = job.delta_prev[moff + i], bp = job.beta_prev[moff + i];
      dg[m] = cn_diag(de, be, rho, r);
      rh[m] = cn_rhs(left, center, right, dp, bp, rho, r);
    }
    if (job.transparent) {
      const double ZERO = 1e-16;
      if (t == 0) {
        double2 o = to_d(u[0]), in = to_d(u[1]);
        if (hypot(in.x, in.y) > ZERO) cn_tbc(o, in, rho, dg[0], rh[0]);
      }
      if (t == T - 1) {
        double2 o = to_d(u[n - 1]), in = to_d(u[n - 2]);
        if (hypot(in.x, in.y) > ZERO) cn_tbc(o, in, rho, dg[M - 1], rh[M - 1]);
      }
    }
    // ---- 2. interior elimination (partition method)
    double2 y[M > 2 ? M - 2 : 1], p[M > 2 ? M - 2 : 1], q[M > 2 ? M - 2 : 1];
    const ReducedRows rr = chunk_eliminate<M>(dg, rh, sub, s0 > 0, s0 + M < n, y, p, q);
    const double2 ea = rr.ea, eb = rr.eb, ec = rr.ec, ed = rr.ed;
    const double2 fa = rr.fa, fb = rr.fb, fc = rr.fc, fd = rr.fd;
    ra[2 * t] = ea; rb[2 * t] = eb; rc[2 * t] = ec; rd[2 * t] = ed;
    ra[2 * t + 1] = fa; rb[2 * t + 1] = fb; rc[2 * t + 1] = fc; rd[2 * t + 1] = fd;
    __syncthreads();
    // ---- 3. reduced system
    cyclic_reduction(ra, rb, rc, rd, nr, t, T);
    // ---- 4. reconstruct
    const double2 xf = rd[2 * t], xl = rd[2 * t + 1];
    const bool save = job.save_every > 0 && saves != nullptr && (step % job.save_every) == 0 &&
                      (step / job.save_every - 1) < job.max_slots;
    C *slot = save ? saves + (long long)(step / job.save_every - 1) * nreal : nullptr;
    double acc = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const C v = from_d<R>(chunk_value<M>(m, xf, xl, y, p, q));
      u[s0 + m] = v;
      if (save && s0 + m < nreal) slot[s0 + m] = v;
      if (flux) flux_add(acc, s0 + m, fw, to_d(v));
    }
    if (flux) flux_warp_total<T>(acc, flux_red[st & 1]);
    __syncthreads();
    if (flux) flux_store<T>(job.flux, step, flux_red[st & 1]);
  }
  for (int i = t; i < nreal; i += T) field[i] = u[i];
}

// Dirichlet ends: the step as one solve.  With A the step's matrix (diagonal
// 1 + i rho/2 + m, off-diagonal s = -i rho/4, m = (beta r + i delta r)/2 at the
// new plane) and m' the old plane's, the right-hand side's matrix is 2 - A +
// (m - m'), so
//   u_new = A^-1 ((2 + m - m') u) - u:
// no stencil, no halo exchange, a pointwise right-hand side (a constant 2 when
// the medium does not change along z).
//
// A is solved from both ends at once (D. J. Evans and M. Hatzopoulos, "A
// parallel linear system solver", Int. J. Comput. Math. 7(3), 1979): with the
// pivots d_i = b_i - s^2/d_(i-1) from the left and e_i = b_i - s^2/e_(i+1) from
// the right,
//   l_i = r_i + hL_i l_(i-1),  hL_i = -s/d_(i-1),
//   p_i = r_i + hR_i p_(i+1),  hR_i = -s/e_(i+1),
//   x_i = w_i (l_i + p_i - r_i),  w_i = 1/(d_i + e_i - b_i).
// The two recurrences are independent: their chains, and the scans that carry
// them across threads, run side by side, where forward and back substitution
// run one after the other.
//
// Thread t of a CTA owns rows t*M .. t*M+M-1 (CTA k of a cluster: k*M*T on).
// A chunk's transfer is y_out = a y_in + b; a depends on the tables only, so
// the scan's levels (Kogge-Stone within a warp, then the warps' totals through
// shared memory, of every CTA of the cluster through distributed shared
// memory) move only b, with the products of a kept per thread:
//   lev  the products a lane's scan levels apply (zero where there is no
//        partner),
//   ex   the product over the warp's chunks before this one in scan order,
//   cf   lane v: the product over the warps between warp v and this one
//        (zero for warps not before it in scan order).
// The totals' buffer alternates between steps, so a step has one barrier.
struct ScanCoef {
  double2 levL[5], levR[5], exL, exR, cfL, cfR;
};

__device__ __forceinline__ double2 shfl_up_d2(double2 v, int d) {
  return mk(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double2 shfl_down_d2(double2 v, int d) {
  return mk(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double2 shfl_xor_d2(double2 v, int d) {
  return mk(__shfl_xor_sync(0xffffffffu, v.x, d), __shfl_xor_sync(0xffffffffu, v.y, d));
}

// The products from each thread's chunk products aL, aR; tot: TW warp totals
// of each direction (shared memory of the calling CTA, gw: this warp's index
// among all TW).  Every thread of the TW warps calls it; publish(w, L, R)
// stores a warp's totals where every warp reads them, sync() follows.
template <int TW, typename Publish, typename Sync>
__device__ __forceinline__ ScanCoef scan_coef(double2 aL, double2 aR, const double2 *tot, int gw,
                                              Publish publish, Sync sync) {
  const int lane = threadIdx.x & 31;
  const double2 zero = mk(0.0, 0.0), one = mk(1.0, 0.0);
  ScanCoef c;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 1 << k;
    const double2 oL = shfl_up_d2(aL, d), oR = shfl_down_d2(aR, d);
    c.levL[k] = lane >= d ? aL : zero;
    c.levR[k] = lane + d < 32 ? aR : zero;
    if (lane >= d) aL = cmul(aL, oL);
    if (lane + d < 32) aR = cmul(aR, oR);
  }
  c.exL = shfl_up_d2(aL, 1);
  if (lane == 0) c.exL = one;
  c.exR = shfl_down_d2(aR, 1);
  if (lane == 31) c.exR = one;
  c.cfL = c.cfR = zero;
  if constexpr (TW > 1) {
    if (lane == 31) publish(gw, 0, aL);
    if (lane == 0) publish(gw, 1, aR);
    sync();
    const int v = lane & (TW - 1);
    if (v < gw) {
      c.cfL = one;
      for (int w = v + 1; w < gw; ++w) c.cfL = cmul(c.cfL, tot[w]);
    }
    if (v > gw) {
      c.cfR = one;
      for (int w = v - 1; w > gw; --w) c.cfR = cmul(c.cfR, tot[TW + w]);
    }
  }
  return c;
}

// Carry-ins of both recurrences from the chunks' ends bL, bR (zero carry-in).
template <int TW, typename Publish, typename Sync>
__device__ __forceinline__ void scan_carry(double2 bL, double2 bR, const ScanCoef &c,
                                           const double2 *tot, int gw, Publish publish, Sync sync,
                                           double2 &cL, double2 &cR) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 1 << k;
    const double2 oL = shfl_up_d2(bL, d), oR = shfl_down_d2(bR, d);
    bL = cfma(c.levL[k], oL, bL);
    bR = cfma(c.levR[k], oR, bR);
  }
  cL = shfl_up_d2(bL, 1);
  cR = shfl_down_d2(bR, 1);
  if (lane == 0) cL = mk(0.0, 0.0);
  if (lane == 31) cR = mk(0.0, 0.0);
  if constexpr (TW > 1) {
    if (lane == 31) publish(gw, 0, bL);
    if (lane == 0) publish(gw, 1, bR);
    sync();
    const int v = lane & (TW - 1);
    double2 sL = cmul(c.cfL, tot[v]), sR = cmul(c.cfR, tot[TW + v]);
#pragma unroll
    for (int d = 1; d < TW; d <<= 1) {
      sL = cadd(sL, shfl_xor_d2(sL, d));
      sR = cadd(sR, shfl_xor_d2(sR, d));
    }
    cL = cfma(c.exL, sL, cL);
    cR = cfma(c.exR, sR, cR);
  }
}

// The solve for the M right-hand sides in r: x replaces r.  hL(m), hR(m),
// w(m): the tables at this thread's row m; coef(): the scan products.
template <int M, int TW, typename TL, typename TR, typename TWt, typename Coef, typename Publish,
          typename Sync, typename Before>
__device__ __forceinline__ void two_sided_solve(double2 (&r)[M], TL hL, TR hR, TWt w,
                                                Coef coef, const double2 *tot, int gw,
                                                Publish publish, Sync sync, Before before_w) {
  double2 acc[M];  // l + p - r
  double2 l = r[0], p = r[M - 1];
#pragma unroll
  for (int k = 0; k < M; ++k) {
    // row k from the left, row M-1-k from the right; an accumulator is set by
    // the first of the two that reaches it
    const int i = k, j = M - 1 - k;
    if (k > 0) l = cfma(hL(i), l, r[i]);
    double2 q = mk(0.0, 0.0);
    if (k > 0) {
      q = cmul(hR(j), p);
      p = cadd(q, r[j]);
    }
    if (i < j) {
      acc[i] = l;
      acc[j] = q;
    } else if (i == j) {
      acc[i] = cadd(l, q);
    } else {
      acc[i] = cadd(acc[i], l);
      acc[j] = cadd(acc[j], q);
    }
  }
  double2 cL, cR;
  scan_carry<TW>(l, p, coef(), tot, gw, publish, sync, cL, cR);
#pragma unroll
  for (int k = 0; k < M; ++k) {
    const int i = k, j = M - 1 - k;
    cL = cmul(hL(i), cL);
    cR = cmul(hR(j), cR);
    acc[i] = cadd(acc[i], cL);
    acc[j] = cadd(acc[j], cR);
  }
  before_w();
#pragma unroll
  for (int m = 0; m < M; ++m) r[m] = cmul(w(m), acc[m]);
}

// The rest of a step: u = x - u, rounded to the field's precision, the save
// and the flux terms of rows s0 ..
template <typename R, int M>
__device__ __forceinline__ double cn_finish(const CnJob &job, int step, double2 (&u)[M],
                                            const double2 (&x)[M], int s0, int nreal, bool flux,
                                            int2 fw) {
  using C = typename Cx<R>::T;
  C *saves = reinterpret_cast<C *>(job.saves);
  const bool save = job.save_every > 0 && saves != nullptr && (step % job.save_every) == 0 &&
                    (step / job.save_every - 1) < job.max_slots;
  C *slot = save ? saves + (long long)(step / job.save_every - 1) * nreal : nullptr;
  double acc = 0.0;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const C v = from_d<R>(csub(x[m], u[m]));
    u[m] = to_d(v);
    if (save && s0 + m < nreal) slot[s0 + m] = v;
    if (flux) flux_add(acc, s0 + m, fw, u[m]);
  }
  return acc;
}

// The flux sum of a step: every warp's total goes to its slot in CTA 0's shared
// memory (part: rows of alternating steps) and one tree adds the slots, so the
// sum does not depend on how many CTAs the problem's warps are spread over.  A
// row is written again only after a later step's scan, whose barrier follows
// its reads.
template <int TW, int K>
__device__ __forceinline__ void cn_flux(const CnJob &job, int step, double acc, double (*part)[TW],
                                        int gw) {
  double *row = part[step & 1];
  const int lane = threadIdx.x & 31;
  double v = acc;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  if constexpr (K == 1) {
    if (lane == 0) row[gw] = v;
    __syncthreads();
  } else {
    cg::cluster_group cluster = cg::this_cluster();
    if (lane == 0) *cluster.map_shared_rank(row + gw, 0) = v;
    cluster.sync();
  }
  if (gw != 0) return;  // the first warp of CTA 0
  v = lane < TW ? row[lane] : 0.0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  if (lane == 0) job.flux.out[step - job.flux.step0] = v;
}

// z-invariant medium: tables and scan products set up once, the field in
// registers for all steps.  K CTAs a problem (a cluster when K > 1).
//
// What bounds it: the latency of two chunk chains and the scan, then its SMs'
// FP64 issue (about 30 operations a row and step).  Measured, us a step, before
// (stencil, then forward and back substitution with (a, b) scans) and now: 256
// rows 1.4 -> 0.53, 1000 2.0 -> 1.0, 2048 2.7 -> 1.40, 4096 4.6 -> 1.42, 16384
// 5.8 -> 2.07; FP32 4096 4.3 -> 1.4, 8192 5.7 -> 2.09.  Against an 80-bit
// Thomas sweep the error after 3000 to 8000 steps fell from 0.1 .. 19e-12 to
// 0.07 .. 6e-12 (12 guides at 1000, 2048 and 4096 rows).
template <typename R, int M, int T, int K, bool FLUX>
__global__ void __launch_bounds__(T) cn_const_kernel(const CnJob *__restrict__ jobs, int step0_ov,
                                                    int nsteps_ov) {
  using C = typename Cx<R>::T;
  constexpr int NC = M * T, W = T / 32, TW = W * K;
  static_assert(T % 32 == 0 && TW <= 32, "whole warps, one lane a warp total");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *sL = reinterpret_cast<double2 *>(smem_raw);  // row m of chunk t at m*T + t
  double2 *sR = sL + NC;
  double2 *sW = sR + NC;
  double2 *tot = sW + NC;  // 2 x 2 x TW
  __shared__ double flux_part[2][TW];
  CnJob job = jobs[blockIdx.x / K];
  if (nsteps_ov >= 0) {
    job.step0 = step0_ov;
    job.nsteps = nsteps_ov;
  }
  const int t = threadIdx.x, rank = K > 1 ? (int)(blockIdx.x % K) : 0;
  const int gw = rank * W + t / 32;
  const int s0 = (rank * T + t) * M;
  // rows nreal .. pad the system (diagonal kCnPad in the tables, zero field)
  const int nreal = job.n_real > 0 ? job.n_real : K * NC;
  const double2 *gL = reinterpret_cast<const double2 *>(job.lu_l) + s0;
  const double2 *gR = reinterpret_cast<const double2 *>(job.lu_r) + s0;
  const double2 *gW = reinterpret_cast<const double2 *>(job.lu_w) + s0;
  double2 aL = mk(1.0, 0.0), aR = mk(1.0, 0.0);
#pragma unroll
  for (int m = 0; m < M; ++m) {
    sL[m * T + t] = gL[m];
    sR[m * T + t] = gR[m];
    sW[m * T + t] = gW[m];
    aL = cmul(aL, gL[m]);
    aR = cmul(aR, gR[m]);
  }
  C *field = reinterpret_cast<C *>(job.field);
  double2 u[M];
#pragma unroll
  for (int m = 0; m < M; ++m) u[m] = s0 + m < nreal ? to_d(field[s0 + m]) : mk(0.0, 0.0);
  int par = 0;
  auto publish = [&](int w, int dir, double2 v) {
    double2 *dst = tot + par * 2 * TW + dir * TW + w;
    if constexpr (K == 1) {
      *dst = v;
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) *cg::this_cluster().map_shared_rank(dst, k) = v;
    }
  };
  auto sync = [] {
    if constexpr (K == 1) __syncthreads();
    else cg::this_cluster().sync();
  };
  if constexpr (K > 1) cg::this_cluster().sync();  // the peers run: their memory may be written
  const ScanCoef c = scan_coef<TW>(aL, aR, tot, gw, publish, sync);
  par = 1;
  for (int st = 0; st < job.nsteps; ++st, par ^= 1) {
    const int step = job.step0 + st;
    int2 fw;
    const bool flux = FLUX && flux_window(job.flux, step, fw);
    double2 x[M];
#pragma unroll
    for (int m = 0; m < M; ++m) x[m] = u[m];
    if (job.two_planes) {
      // (2 + m - m') u, the 2 being in the tables
#pragma unroll
      for (int m = 0; m < M; ++m)
        if (s0 + m < nreal) {
          const double2 h = mk(0.25 * job.r * (job.beta[s0 + m] - job.beta_prev[s0 + m]),
                               0.25 * job.r * (job.delta[s0 + m] - job.delta_prev[s0 + m]));
          x[m] = cfma(h, u[m], u[m]);
        }
    }
    two_sided_solve<M, TW>(
        x, [&](int m) { return sL[m * T + t]; }, [&](int m) { return sR[m * T + t]; },
        [&](int m) { return sW[m * T + t]; }, [&]() -> const ScanCoef & { return c; },
        tot + par * 2 * TW, gw, publish, sync, [] {});
    const double acc = cn_finish<R>(job, step, u, x, s0, nreal, flux, fw);
    if constexpr (FLUX)
      if (flux) cn_flux<TW, K>(job, step, acc, flux_part, gw);
  }
  if constexpr (K > 1) cg::this_cluster().sync();  // no CTA leaves while a peer writes to it
#pragma unroll
  for (int m = 0; m < M; ++m)
    if (s0 + m < nreal) field[s0 + m] = from_d<R>(u[m]);
}

// Media sampled per step: every step has its own matrix, but none depends on
// the field, so a window of steps is factored ahead (cn_pivot_kernel,
// cn_table_kernel) and the sequential kernel (cn_planes_kernel) only solves with
// its tables.  A launch takes a list of problems (CnPlanes); every problem's
// arithmetic is the same alone and among others, and whatever the windows.
//
// Tables of a step: [c | hL | hR | w], c = 2 + m - m', rows in the solving
// kernel's order (row m of thread tt at m*TT + tt, TT threads over the
// cluster), then the 14 scan products of each thread.
constexpr int kCnCoefs = 14;
__host__ __device__ constexpr size_t cn_step_entries(int M, int TT) {
  return (size_t)TT * (4 * M + kCnCoefs);
}

// Inverse of a pivot as an unevaluated sum hi + lo.
struct PivotInv {
  double2 hi, lo;
};

// 1 / (b + q^2 prev), prev an inverse pivot: the sum and the reciprocal carry
// a second word each (two-sum and FMA residuals, T. J. Dekker, "A
// floating-point technique for extending the available precision", Numer.
// Math. 18, 1971; one Newton step from the rounded reciprocal).  Rounded
// pivots would err the same way at every row of a uniform stretch and at every
// step.
struct QSq {
  double hi, lo;
};
__device__ __forceinline__ void pivot_sum(double b, QSq q2, double hi, double lo, double &s, double &t) {
  const double p = __dmul_rn(q2.hi, hi);
  const double e = __fma_rn(q2.hi, hi, -p) + __fma_rn(q2.hi, lo, __dmul_rn(q2.lo, hi));
  s = __dadd_rn(b, p);
  const double bb = __dsub_rn(s, b);
  t = __dadd_rn(__dadd_rn(__dsub_rn(b, __dsub_rn(s, bb)), __dsub_rn(p, bb)), e);
}
// 1 / (d + dl), dl the second word of d.
__device__ __forceinline__ PivotInv inverse_words(double2 d, double2 dl) {
  const double2 r = crecip(d);
  // residual 1 - (d + dl) r
  const double p1 = __dmul_rn(d.x, r.x), p2 = __dmul_rn(d.y, r.y);
  const double e1 = __fma_rn(d.x, r.x, -p1), e2 = __fma_rn(d.y, r.y, -p2);
  const double u = __dsub_rn(1.0, p1);  // exact or small: p1 - p2 is 1 to rounding
  const double v = __dadd_rn(u, p2), vb = __dsub_rn(v, u);
  const double ve = __dadd_rn(__dsub_rn(u, __dsub_rn(v, vb)), __dsub_rn(p2, vb));
  const double ub = __dsub_rn(1.0, u), ue = __dsub_rn(ub, p1);
  const double rx = v + (ve + ue - e1 + e2) - (dl.x * r.x - dl.y * r.y);
  const double p3 = __dmul_rn(d.x, r.y), p4 = __dmul_rn(d.y, r.x);
  const double ry = -(p3 + p4) - (__fma_rn(d.x, r.y, -p3) + __fma_rn(d.y, r.x, -p4)) -
                    (dl.x * r.y + dl.y * r.x);
  return {r, cmul(r, mk(rx, ry))};
}
__device__ __forceinline__ PivotInv pivot_inverse(double2 b, QSq q2, PivotInv prev) {
  double2 d, dl;
  pivot_sum(b.x, q2, prev.hi.x, prev.lo.x, d.x, dl.x);
  pivot_sum(b.y, q2, prev.hi.y, prev.lo.y, d.y, dl.y);
  return inverse_words(d, dl);
}

// hi + lo rounded to one word, up or down by a draw of 32 bits with probabilities
// that make the mean exact (G. E. Forsythe, "Round-off errors in numerical
// integration on automatic machinery", Bull. AMS 56, 1950).  Rounded to
// nearest, a table entry errs the same way at every row of a uniform stretch and
// at every step, and the errors of a pass add up; this way they do not.
__device__ __forceinline__ double round_dithered(double hi, double lo, unsigned draw) {
  const double s = __dadd_rn(hi, lo), t = __dsub_rn(lo, __dsub_rn(s, hi));
  const double top = __longlong_as_double(__double_as_longlong(s) & 0x7ff0000000000000ll);
  // the draw, -1/2 .. 1/2 units in the last place of s
  return __dadd_rn(s, __fma_rn((double)(int)draw * 5.1698788284564230e-26, top, t));
}
// A draw for entry k of a step: the finalizer of MurmurHash3 (A. Appleby, public
// domain) over both.
__device__ __forceinline__ unsigned dither(unsigned step, unsigned k) {
  unsigned h = step * 0x9e3779b1u + k;
  h ^= h >> 16;
  h *= 0x85ebca6bu;
  h ^= h >> 13;
  h *= 0xc2b2ae35u;
  return h ^ (h >> 16);
}

// Pivots of one recurrence of a step: row k (from the left, or DIR < 0 from the
// right) from de[k * DIR] and be[k * DIR] to hi[k * DIR] and lo[k * DIR].
template <int DIR>
__device__ __forceinline__ void pivot_chain(const double *__restrict__ de, const double *__restrict__ be,
                                            double2 *__restrict__ hi, float2 *__restrict__ lo, int n,
                                            double rho, double r) {
  const double q = 0.25 * rho;
  QSq q2;
  q2.hi = __dmul_rn(q, q);
  q2.lo = __fma_rn(q, q, -q2.hi);
  PivotInv inv = {mk(0.0, 0.0), mk(0.0, 0.0)};
  auto row = [&](int k, double d, double b) {
    inv = pivot_inverse(cn_diag(d, b, rho, r), q2, inv);
    hi[k * DIR] = inv.hi;
    lo[k * DIR] = make_float2((float)inv.lo.x, (float)inv.lo.y);
  };
  // whole groups of rows, each group's inputs loaded while the one before is
  // worked on
  constexpr int U = 8;
  double dn[U], bn[U];
  const int full = n / U;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    dn[u] = full > 0 ? de[u * DIR] : 0.0;
    bn[u] = full > 0 ? be[u * DIR] : 0.0;
  }
#pragma unroll 1
  for (int g = 0; g < full; ++g) {
    double d[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      d[u] = dn[u];
      b[u] = bn[u];
    }
    const int next = g + 1 < full ? U : 0;  // the last group loads itself again
#pragma unroll
    for (int u = 0; u < U; ++u) {
      dn[u] = de[(next + u) * DIR];
      bn[u] = be[(next + u) * DIR];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) row(u, d[u], b[u]);
    de += U * DIR;
    be += U * DIR;
    hi += U * DIR;
    lo += U * DIR;
  }
#pragma unroll 1
  for (int k = 0; k < n - full * U; ++k) row(k, de[k * DIR], be[k * DIR]);
}

// The pivots of a window's steps: the two recurrences of a step are serial (some
// 130 ns a row), so a thread takes one of them and a warp 32 steps'; a window of
// a few hundred steps then needs some twenty warps, and problems stepping side by
// side share the SMs.  Pivot i of step st and direction d goes to workspace
// entry (2 st + d) * np + i, second words after the first ones.
__global__ void __launch_bounds__(32)
    cn_pivot_kernel(const CnJob *__restrict__ jobs, const CnPlanes *__restrict__ list, const CnPlanes one,
                    int np) {
  const CnPlanes w = list ? list[blockIdx.y] : one;
  const int dir = blockIdx.x & 1, st = (blockIdx.x >> 1) * 32 + threadIdx.x;
  if (!w.factor || st >= w.count) return;
  const CnJob &job = jobs[blockIdx.y];
  const int n = job.n_real > 0 ? job.n_real : np;
  const long long off = job.mat_stride * (long long)(w.first + st - job.mat_step0);
  const double *de = job.delta + off, *be = job.beta + off;
  const size_t at = (size_t)(2 * st + dir) * np;
  double2 *hi = w.pivots + at;
  float2 *lo = reinterpret_cast<float2 *>(w.pivots + 2 * (size_t)w.count * np) + at;
  if (dir == 0) pivot_chain<1>(de, be, hi, lo, n, job.rho, job.r);
  else pivot_chain<-1>(de + n - 1, be + n - 1, hi + n - 1, lo + n - 1, n, job.rho, job.r);
}

// The tables of a window's steps from its pivots, a CTA a step; everything here
// is parallel over rows.
template <int M, int TT>
__global__ void __launch_bounds__(TT)
    cn_table_kernel(const CnJob *__restrict__ jobs, const CnPlanes *__restrict__ list, const CnPlanes one) {
  constexpr int NP = M * TT, TW = TT / 32;
  __shared__ double2 tot[2 * TW];
  const CnPlanes pw = list ? list[blockIdx.y] : one;
  const int st = blockIdx.x;
  if (!pw.factor || st >= pw.count) return;
  const CnJob job = jobs[blockIdx.y];
  const int t = threadIdx.x, n = job.n_real > 0 ? job.n_real : NP;
  const long long off = job.mat_stride * (long long)(pw.first + st - job.mat_step0);
  const double *de = job.delta + off, *be = job.beta + off;
  const double *dp = job.delta_prev + off, *bp = job.beta_prev + off;
  const double2 *hi = pw.pivots + (size_t)(2 * st) * NP;
  const float2 *lo =
      reinterpret_cast<const float2 *>(pw.pivots + 2 * (size_t)pw.count * NP) + (size_t)(2 * st) * NP;
  // the padding rows' pivots are kCnPad; beyond the system there is none
  auto pivot = [&](int dir, int i) {
    const double2 zero = mk(0.0, 0.0);
    if (i < 0 || i >= NP) return PivotInv{zero, zero};
    if (i >= n) return PivotInv{mk(1.0 / kCnPad, 0.0), zero};
    return PivotInv{hi[dir * NP + i], to_d(lo[dir * NP + i])};
  };
  const double q = 0.25 * job.rho;
  QSq q2;
  q2.hi = __dmul_rn(q, q);
  q2.lo = __fma_rn(q, q, -q2.hi);
  auto draw = [step = pw.first + st](int row, int k) { return dither((unsigned)step, (unsigned)row * 8u + k); };
  double2 *out = pw.tabs + st * cn_step_entries(M, TT);
  double2 aL = mk(1.0, 0.0), aR = mk(1.0, 0.0);
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int i = t * M + m;
    const PivotInv il = pivot(0, i - 1), ir = pivot(1, i + 1);
    // i q / pivot
    auto off = [q](double hi, double lo, unsigned d) {
      const double p = __dmul_rn(q, hi);
      return round_dithered(p, __fma_rn(q, lo, __fma_rn(q, hi, -p)), d);
    };
    const double2 hL = mk(-off(il.hi.y, il.lo.y, draw(i, 0)), off(il.hi.x, il.lo.x, draw(i, 1)));
    const double2 hR = mk(-off(ir.hi.y, ir.lo.y, draw(i, 2)), off(ir.hi.x, ir.lo.x, draw(i, 3)));
    double2 c = mk(2.0, 0.0), b = mk(kCnPad, 0.0);
    if (i < n) {
      b = cn_diag(de[i], be[i], job.rho, job.r);
      c = mk(fma(0.5 * job.r, be[i] - bp[i], 2.0), 0.5 * job.r * (de[i] - dp[i]));
    }
    // d + e - b = b + q^2 (1/d' + 1/e'), d' and e' the neighbouring pivots
    double2 d, dl, f, fl;
    pivot_sum(b.x, q2, il.hi.x, il.lo.x, d.x, dl.x);
    pivot_sum(b.y, q2, il.hi.y, il.lo.y, d.y, dl.y);
    pivot_sum(d.x, q2, ir.hi.x, ir.lo.x, f.x, fl.x);
    pivot_sum(d.y, q2, ir.hi.y, ir.lo.y, f.y, fl.y);
    const PivotInv wi = inverse_words(f, mk(fl.x + dl.x, fl.y + dl.y));
    const double2 w = mk(round_dithered(wi.hi.x, wi.lo.x, draw(i, 4)),
                         round_dithered(wi.hi.y, wi.lo.y, draw(i, 5)));
    out[m * TT + t] = c;
    out[(M + m) * TT + t] = hL;
    out[(2 * M + m) * TT + t] = hR;
    out[(3 * M + m) * TT + t] = w;
    aL = cmul(aL, hL);
    aR = cmul(aR, hR);
  }
  const ScanCoef c = scan_coef<TW>(
      aL, aR, tot, t / 32, [&](int w, int dir, double2 v) { tot[dir * TW + w] = v; },
      [] { __syncthreads(); });
  double2 *oc = out + 4 * NP;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    oc[k * TT + t] = c.levL[k];
    oc[(5 + k) * TT + t] = c.levR[k];
  }
  oc[10 * TT + t] = c.exL;
  oc[11 * TT + t] = c.exR;
  oc[12 * TT + t] = c.cfL;
  oc[13 * TT + t] = c.cfR;
}

__device__ __forceinline__ void cn_cp_async16(double2 *dst, const double2 *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cn_cp_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N> __device__ __forceinline__ void cn_cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

constexpr bool cn_c_in_registers(int M, int T) { return M * T > 1024; }

// The steps of a window with the tables above.  Every thread copies its own
// table entries a step ahead into slots of its own (no barrier): hL and hR,
// used until the carries are folded in, into alternating buffers, the others
// into the slots just read.  Four copy groups a step, in the order they are
// used: {hL, hR}, {c}, {products}, {w}.  With 2048 rows a CTA there is no room
// for c, which waits in registers (slower elsewhere: 200 rows, 400 steps 719
// against 590 us).
// What bounds it: the const kernel's chains plus the tables' way from L2 (92
// bytes a row and step into its SMs), and the pivot chains in front of every
// window.  Measured, us a step and us of pivots a window (step by step,
// cn_kernel): 300 rows 1.0 and 75 (8.2), 1000: 1.2 and 157 (10.8), 1501: 1.9 and
// 218 (15.1), 4000: 1.9 and 513 (27); eight problems of 1501 rows and 200 steps
// in a batch 0.75 ms (3.1), 48 of them 1.8 (3.1).  Errors against an 80-bit sweep after
// 300 steps, the median of three guides (step by step; with entries rounded to
// nearest): 64 rows 4e-15 (6e-15; 4e-14), 128: 3e-15 (9e-15; 2e-14), 300: 3e-15
// (6e-15; 2e-14), 1000: 1.4e-14 (3e-14; 5e-14), 3000: 2e-14 (2e-12; 9e-14); with
// pivots of one word 1501 and 3000 rows 1.4e-12 and 2.2e-12.
template <typename R, int M, int T, int K, bool FLUX>
__global__ void __launch_bounds__(T) cn_planes_kernel(const CnJob *__restrict__ jobs,
                                                     const CnPlanes *__restrict__ list,
                                                     const CnPlanes one) {
  using C = typename Cx<R>::T;
  constexpr int NC = M * T, W = T / 32, TW = W * K, TT = T * K;
  constexpr bool CREG = cn_c_in_registers(M, T);
  constexpr int AHEAD = CREG ? 2 : 3;  // groups younger than the one to wait for
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *sH = reinterpret_cast<double2 *>(smem_raw);  // 2 x [hL | hR]
  double2 *sC = sH + 4 * NC;
  double2 *sW = CREG ? sC : sC + NC;
  double2 *sP = sW + NC;             // 14 x T
  double2 *tot = sP + kCnCoefs * T;  // 2 x 2 x TW
  __shared__ double flux_part[2][TW];
  const CnPlanes pw = list ? list[blockIdx.x / K] : one;
  const int step0 = pw.step0, nsteps = pw.nsteps;
  if (nsteps <= 0) return;  // the whole cluster
  const CnJob job = jobs[blockIdx.x / K];
  const double2 *tabs = pw.tabs + (step0 - pw.first) * cn_step_entries(M, T * K);
  const int t = threadIdx.x, rank = K > 1 ? (int)(blockIdx.x % K) : 0;
  const int gw = rank * W + t / 32, tt = rank * T + t;
  const int s0 = tt * M;
  const int nreal = job.n_real > 0 ? job.n_real : K * NC;
  auto fetch = [&](int st, int table, double2 *dst, int rows) {  // rows of one table
    if (st < nsteps) {
      const double2 *src = tabs + st * cn_step_entries(M, TT) + (size_t)table * M * TT + tt;
#pragma unroll
      for (int m = 0; m < rows; ++m) cn_cp_async16(dst + m * T + t, src + (size_t)m * TT);
    }
  };
  auto fetch_h = [&](int st) {
    double2 *dst = sH + (st & 1) * 2 * NC;
    fetch(st, 1, dst, M);
    fetch(st, 2, dst + NC, M);
    cn_cp_commit();
  };
  double2 c[CREG ? M : 1];
  auto fetch_c = [&](int st) {
    if constexpr (!CREG) {
      fetch(st, 0, sC, M);
      cn_cp_commit();
    } else if (st < nsteps) {
#pragma unroll
      for (int m = 0; m < M; ++m) c[m] = __ldg(tabs + st * cn_step_entries(M, TT) + (size_t)m * TT + tt);
    }
  };
  auto fetch_p = [&](int st) { fetch(st, 4, sP, kCnCoefs); cn_cp_commit(); };
  auto fetch_w = [&](int st) { fetch(st, 3, sW, M); cn_cp_commit(); };
  fetch_h(0);
  fetch_c(0);
  fetch_p(0);
  fetch_w(0);
  C *field = reinterpret_cast<C *>(job.field);
  double2 u[M];
#pragma unroll
  for (int m = 0; m < M; ++m) u[m] = s0 + m < nreal ? to_d(field[s0 + m]) : mk(0.0, 0.0);
  int par = 0;
  auto publish = [&](int w, int dir, double2 v) {
    double2 *dst = tot + par * 2 * TW + dir * TW + w;
    if constexpr (K == 1) {
      *dst = v;
    } else {
#pragma unroll
      for (int k = 0; k < K; ++k) *cg::this_cluster().map_shared_rank(dst, k) = v;
    }
  };
  auto sync = [] {
    if constexpr (K == 1) __syncthreads();
    else cg::this_cluster().sync();
  };
  if constexpr (K > 1) cg::this_cluster().sync();  // the peers run: their memory may be written
  for (int st = 0; st < nsteps; ++st, par ^= 1) {
    const int step = step0 + st;
    int2 fw;
    const bool flux = FLUX && flux_window(job.flux, step, fw);
    cn_cp_wait<2>();  // {hL, hR} and {c} of this step
    fetch_h(st + 1);
    const double2 *hl = sH + (st & 1) * 2 * NC + t, *hr = hl + NC;
    double2 x[M];
#pragma unroll
    for (int m = 0; m < M; ++m) x[m] = cmul(CREG ? c[m] : sC[m * T + t], u[m]);
    fetch_c(st + 1);
    two_sided_solve<M, TW>(
        x, [&](int m) { return hl[m * T]; }, [&](int m) { return hr[m * T]; },
        [&](int m) { return sW[m * T + t]; },
        [&] {
          cn_cp_wait<AHEAD>();
          ScanCoef c;
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            c.levL[k] = sP[k * T + t];
            c.levR[k] = sP[(5 + k) * T + t];
          }
          c.exL = sP[10 * T + t];
          c.exR = sP[11 * T + t];
          c.cfL = sP[12 * T + t];
          c.cfR = sP[13 * T + t];
          return c;
        },
        tot + par * 2 * TW, gw, publish, sync, [&] {
          fetch_p(st + 1);
          cn_cp_wait<AHEAD>();  // {w}
        });
    fetch_w(st + 1);
    const double acc = cn_finish<R>(job, step, u, x, s0, nreal, flux, fw);
    if constexpr (FLUX)
      if (flux) cn_flux<TW, K>(job, step, acc, flux_part, gw);
  }
  cn_cp_wait<0>();
  if constexpr (K > 1) cg::this_cluster().sync();  // no CTA leaves while a peer writes to it
#pragma unroll
  for (int m = 0; m < M; ++m)
    if (s0 + m < nreal) field[s0 + m] = from_d<R>(u[m]);
}

static constexpr int kCnM = 8;

template <typename K_, typename... A>
static cudaError_t cn_cluster_launch(K_ kernel, int ctas, int cluster, int threads, size_t smem,
                                     cudaStream_t s, A... args) {
  const cudaError_t e = raise_dynamic_smem((const void *)kernel, (int)smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename R, int M, int T, int K>
static cudaError_t cn_const_launch_t(const CnJob *d_jobs, int nj, int step0, int nsteps,
                                     cudaStream_t s, bool flux) {
  constexpr size_t smem = sizeof(double2) * (3 * M * T + 4 * (T / 32) * K);
  return flux ? cn_cluster_launch(cn_const_kernel<R, M, T, K, true>, nj * K, K, T, smem, s, d_jobs,
                                  step0, nsteps)
              : cn_cluster_launch(cn_const_kernel<R, M, T, K, false>, nj * K, K, T, smem, s, d_jobs,
                                  step0, nsteps);
}

bool cn_const_supported(Precision, int n) {
  return n >= 8 * kCnM && !(n & (n - 1)) && n <= 16384;
}

// Rows a thread, threads a CTA and CTAs a problem.  From 4096 rows on a
// problem alone is faster on more SMs (4096: 3.0 us a step on one, 1.72 on
// two, 1.42 on four; 8192 in FP32: 2.93 on two, 2.09 on four; 16384: 2.79 on
// four, 2.07 on eight), at more SM time a problem.  The widest form runs for
// which every problem of the launch finds its SMs free beside the `others` that
// the caller's other handles with work enqueued may be using: an SM for each of a
// 2-D kind, all of them for one of a 3-D kind.  (A 1024^2 ADI half step is one wave of 147
// CTAs, an SM each: beside a problem on four SMs it takes two waves, 40 us a
// step against 22.9.)  The forms have the same chunks and warps and give the
// same bits.  2048 rows gain too little (1.40 on one SM, 1.31 on two).
constexpr int kSms = 148;
static bool cn_wide(int nj, int ctas, int others) {
  // PXP_CN_CLUSTER=0|1 pins the narrowest or the widest form
  const char *pin = std::getenv("PXP_CN_CLUSTER");
  if (pin && (pin[0] == '0' || pin[0] == '1')) return pin[0] == '1';
  return (long long)nj * ctas + others <= kSms;
}
cudaError_t launch_cn_const(Precision p, const CnJob *d_jobs, int nj, int n, int step0, int nsteps,
                            cudaStream_t s, bool flux, int others) {
  if (nj <= 0) return cudaSuccess;
  auto wide = [&](int ctas) { return cn_wide(nj, ctas, others); };
#define PXP_CT(MM, TT, KK)                                                                \
  p == kFP64 ? cn_const_launch_t<double, MM, TT, KK>(d_jobs, nj, step0, nsteps, s, flux) \
             : cn_const_launch_t<float, MM, TT, KK>(d_jobs, nj, step0, nsteps, s, flux)
  switch (n) {
    case 64: return PXP_CT(2, 32, 1);
    case 128: return PXP_CT(4, 32, 1);
    case 256: return PXP_CT(8, 32, 1);
    case 512: return PXP_CT(8, 64, 1);
    case 1024: return PXP_CT(8, 128, 1);
    case 2048: return PXP_CT(16, 128, 1);
    case 4096: return wide(4) ? PXP_CT(8, 128, 4) : wide(2) ? PXP_CT(8, 256, 2) : PXP_CT(8, 512, 1);
    case 8192: return wide(4) ? PXP_CT(16, 128, 4) : PXP_CT(16, 256, 2);
    case 16384: return wide(8) ? PXP_CT(16, 128, 8) : PXP_CT(16, 256, 4);
    default: return cudaErrorInvalidValue;
  }
#undef PXP_CT
}

template <int M, int TT>
static cudaError_t cn_factor_launch_t(const CnJob *d_jobs, const CnPlanes *d_list, const CnPlanes &one,
                                      int nj, int count, cudaStream_t s) {
  cn_pivot_kernel<<<dim3(2 * ((count + 31) / 32), nj), 32, 0, s>>>(d_jobs, d_list, one, M * TT);
  cn_table_kernel<M, TT><<<dim3(count, nj), TT, 0, s>>>(d_jobs, d_list, one);
  return cudaGetLastError();
}

template <typename R, int M, int T, int K>
static cudaError_t cn_planes_launch_t(const CnJob *d_jobs, const CnPlanes *d_list, const CnPlanes &one,
                                      int nj, cudaStream_t s, bool flux) {
  constexpr size_t smem =
      sizeof(double2) * ((cn_c_in_registers(M, T) ? 5 : 6) * M * T + kCnCoefs * T + 4 * (T / 32) * K);
  static_assert(smem <= 226 * 1024, "tables exceed shared memory");
  return flux ? cn_cluster_launch(cn_planes_kernel<R, M, T, K, true>, nj * K, K, T, smem, s, d_jobs, d_list,
                                  one)
              : cn_cluster_launch(cn_planes_kernel<R, M, T, K, false>, nj * K, K, T, smem, s, d_jobs, d_list,
                                  one);
}

// By the medium, not by a call's steps, so that a problem takes one path
// however its steps are split.  Below some 20 steps the pivots cost more than
// the faster steps save (us for 16 and 24 steps in one call, step by step and
// here: 100 rows 98, 137 and 56, 64; 300: 150, 215 and 90, 98; 1000: 194, 280 and
// 177, 186; 1501: 262, 383 and 249, 264; 4000: 456, 672 and 545, 559).
bool cn_planes_supported(int n, int planes) { return n >= 64 && n <= 4096 && planes >= 24; }

// The tables spread a problem's work over SMs that a single one leaves idle; many
// problems side by side fill the SMs anyway, and theirs go through HBM (280 bytes a
// row and step).  Measured with 200 steps in a batch, ms step by step and with
// tables: 250 rows, 148 problems 1.34 and 1.28; 500 rows, 96: 1.83 and 1.40, 148:
// 1.85 and 2.20; 1000 rows, 96: 2.30 and 2.12, 148: 2.33 and 3.30; 1501 rows, 80:
// 3.13 and 2.90, 96: 3.13 and 3.26, 148: 3.16 and 5.03; 2048 rows, 64: 3.30 and
// 2.84, 80: 3.32 and 3.63; 4000 rows, 48: 5.50 and 4.95, 64: 5.51 and 6.89, 148:
// 5.54 and 11.8.
bool cn_planes_pay(int n, int nj) {
  return nj <= (n <= 256 ? 148 : n <= 512 ? 120 : n <= 1024 ? 100 : n <= 2048 ? 72 : 48);
}

// Chunk and threads of a problem of n padded rows (64 .. 4096).
static void cn_planes_shape(int n, int *m, int *tt) {
  *tt = n < 256 ? 32 : n / 8;
  *m = n / *tt;
}
size_t cn_table_bytes(int n) {
  int m, tt;
  cn_planes_shape(n, &m, &tt);
  return sizeof(double2) * cn_step_entries(m, tt);
}
size_t cn_pivot_bytes(int n) { return 2 * (sizeof(double2) + sizeof(float2)) * (size_t)n; }

cudaError_t launch_cn_factor(const CnJob *d_jobs, const CnPlanes *d_list, const CnPlanes &one, int nj,
                             int count, int n, cudaStream_t s) {
  if (nj <= 0 || count <= 0) return cudaSuccess;
#define PXP_CF(NN, MM, TT) case NN: return cn_factor_launch_t<MM, TT>(d_jobs, d_list, one, nj, count, s);
  switch (n) {
    PXP_CF(64, 2, 32) PXP_CF(128, 4, 32) PXP_CF(256, 8, 32) PXP_CF(512, 8, 64) PXP_CF(1024, 8, 128)
    PXP_CF(2048, 8, 256) PXP_CF(4096, 8, 512)
    default: return cudaErrorInvalidValue;
  }
#undef PXP_CF
}

// CTAs a problem by the same rule as launch_cn_const's.
cudaError_t launch_cn_planes(Precision p, const CnJob *d_jobs, const CnPlanes *d_list, const CnPlanes &one,
                             int nj, int n, cudaStream_t s, bool flux, int others) {
  if (nj <= 0) return cudaSuccess;
#define PXP_CP(MM, TT, KK)                                                                  \
  p == kFP64 ? cn_planes_launch_t<double, MM, TT, KK>(d_jobs, d_list, one, nj, s, flux)     \
             : cn_planes_launch_t<float, MM, TT, KK>(d_jobs, d_list, one, nj, s, flux)
  switch (n) {
    case 64: return PXP_CP(2, 32, 1);
    case 128: return PXP_CP(4, 32, 1);
    case 256: return PXP_CP(8, 32, 1);
    case 512: return PXP_CP(8, 64, 1);
    case 1024: return PXP_CP(8, 128, 1);
    case 2048: return cn_wide(nj, 2, others) ? PXP_CP(8, 128, 2) : PXP_CP(8, 256, 1);
    case 4096: return cn_wide(nj, 4, others) ? PXP_CP(8, 128, 4) : PXP_CP(8, 256, 2);
    default: return cudaErrorInvalidValue;
  }
#undef PXP_CP
}

template <typename R, int T, bool FLUX>
static cudaError_t cn_launch_f(const CnJob *d_jobs, int nj, int step0, int nsteps,
                               cudaStream_t s) {
  using C = typename Cx<R>::T;
  size_t smem = sizeof(double2) * 4 * 2 * T + sizeof(C) * kCnM * T;
  auto k = cn_kernel<R, kCnM, T, FLUX>;
  {  // the static flux slots count against the 48 KB default too
    const cudaError_t attr = raise_dynamic_smem((const void *)k, (int)smem);
    if (attr != cudaSuccess) return attr;
  }
  k<<<nj, T, smem, s>>>(d_jobs, step0, nsteps);
  return cudaGetLastError();
}

template <typename R, int T>
static cudaError_t cn_launch_t(const CnJob *d_jobs, int nj, int step0, int nsteps, cudaStream_t s,
                               bool flux) {
  return flux ? cn_launch_f<R, T, true>(d_jobs, nj, step0, nsteps, s)
              : cn_launch_f<R, T, false>(d_jobs, nj, step0, nsteps, s);
}

int cn_padded_n(int n) {
  int t = 2;
  while (t * kCnM < n) t *= 2;
  return t * kCnM;
}

bool cn_supported(Precision p, int n) {
  if (n < 2 * kCnM) return false;
  const int np = cn_padded_n(n);
  return p == kFP64 ? np <= 4096 : np <= 8192;
}

cudaError_t launch_cn(Precision p, const CnJob *d_jobs, int nj, int n, int step0, int nsteps,
                      cudaStream_t s, bool flux) {
  if (nj <= 0) return cudaSuccess;
  const int T = n / kCnM;
#define PXP_CN(TT)                                                                 \
  case TT:                                                                         \
    return p == kFP64 ? cn_launch_t<double, TT>(d_jobs, nj, step0, nsteps, s, flux) \
                      : cn_launch_t<float, TT>(d_jobs, nj, step0, nsteps, s, flux);
  switch (T) {
    PXP_CN(2) PXP_CN(4) PXP_CN(8) PXP_CN(16) PXP_CN(32) PXP_CN(64) PXP_CN(128) PXP_CN(256)
    PXP_CN(512)
    case 1024:
      if (p == kFP32) return cn_launch_t<float, 1024>(d_jobs, nj, step0, nsteps, s, flux);
      return cudaErrorInvalidValue;
    default:
      return cudaErrorInvalidValue;
  }
#undef PXP_CN
}

}  // namespace pxp
