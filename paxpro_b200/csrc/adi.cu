// adi.cu -- K-ADI: one alternating-direction half step with the right-hand
// side stencil fused with a parallel complex tridiagonal solve.
//
// Replaces ADI::xImplicit / ADI::yImplicit / ADI::applyTBC
// (src/alternatingDirectionSolver.cpp:8-234) and the ThomasAlgorithm sweep
// over the chain of n*n unknowns (include/thomasAlgorithm.tpp:2-32), whose
// zero sub-diagonal entries at every system start make the n systems of a
// half step independent.
//
// A CTA owns G consecutive systems.  It stages them, plus one halo system on
// each side for the explicit stencil, in shared memory with loads that are
// coalesced for either layout (systems interleaved in memory for the x half
// step, contiguous for the y half step).  Each system is split into chunks,
// one per thread; the diagonals are built with the reference's operation
// order (matrix coefficients equal the reference's), the chunk interior is
// eliminated in registers, and the reduced system, one unknown a chunk, is
// solved by parallel cyclic reduction.  The solution goes back through shared
// memory for coalesced stores.
//
// Materials: a first-hit sphere list evaluated per point with rounded FP64
// operations (the same r^2 < R^2 test as the oracle); the host culls, per
// half step, spheres whose dz^2 alone is >= R^2, which cannot contain any
// point of the plane.
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "bulk_copy.cuh"
#include "csg.cuh"
#include "pxp_complex.cuh"
#include "pxp_kernels.h"
#include "scan_solve.cuh"

namespace pxp {

// The material of the half step's plane at (x, y); idx: the point's index in
// the field's layout, for a sampled plane.
__device__ __forceinline__ void sphere_material(const AdiHalf &h, double x, double y,
                                                long long idx, double &delta, double &beta) {
  if (h.plane_delta) {
    delta = opaque(h.plane_delta[idx]);
    beta = opaque(h.plane_beta[idx]);
    return;
  }
  if (h.csg.active) {
    csg_material(h.csg, x, y, h.z, delta, beta);
    return;
  }
  delta = 0.0;
  beta = 0.0;
  const int n = h.nspheres;
  const Sphere *list = n > kInlineSpheres ? h.spheres_all : h.spheres;
  for (int i = 0; i < n; ++i) {
    const Sphere sp = list[i];
    double ddx = __dsub_rn(x, sp.cx), ddy = __dsub_rn(y, sp.cy), ddz = __dsub_rn(h.z, sp.cz);
    double rsq = __dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)), __dmul_rn(ddz, ddz));
    if (rsq < __dmul_rn(sp.r, sp.r)) {
      delta = sp.delta;
      beta = sp.beta;
      return;
    }
  }
}

// Transparent-boundary factor 0.5*i*exp(i*kd)/kd2 with kd = -i*log(ratio),
// Re(kd) clamped at 0 (src/alternatingDirectionSolver.cpp:157-234).
__device__ __forceinline__ double2 tbc_factor(double2 num, double2 den) {
  double2 ratio = cx_div_rn(num, den);
  double2 lg = mk(log(hypot(ratio.x, ratio.y)), atan2(ratio.y, ratio.x));
  double2 kd = cx_mul_rn(mk(-0.0, -1.0), lg);
  if (kd.x < 0.0) kd.x = 0.0;
  double2 ik = cx_mul_rn(mk(0.0, 1.0), kd);
  double e = exp(ik.x), sn, cs;
  sincos(ik.y, &sn, &cs);
  return cx_mul_rn(mk(0.0, 0.5), mk(e * cs, e * sn));
}

// Diagonal of the rows that pad a system to whole chunks.
constexpr double kAdiPad = 1e30;

__device__ __forceinline__ void group_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(count) : "memory");
}

// Diagonal of the row at (x, y), from the plane's material there.
__device__ __forceinline__ double2 adi_diag(const AdiHalf &h, double x, double y, long long idx,
                                            double inv_impl) {
  double delta, beta;
  sphere_material(h, x, y, idx, delta, beta);
  if (!h.y_implicit)  // 1.0/dz + i/(k dx dx) + beta*k + i*delta*k   (reference :38)
    return mk(__dadd_rn(h.inv_dzh, __dmul_rn(beta, h.k)), __dadd_rn(inv_impl, __dmul_rn(delta, h.k)));
  // 1.0/dz + i/(k dy dy + beta*k + i*delta*k)   (reference :103, as written);
  // in vacuum i/(k dy dy) exactly
  double2 d = mk(0.0, inv_impl);
  if (delta != 0.0 || beta != 0.0)
    d = cx_div_rn(mk(0.0, 1.0),
                  mk(__dadd_rn(h.kd2_impl, __dmul_rn(beta, h.k)), __dmul_rn(delta, h.k)));
  return mk(__dadd_rn(d.x, h.inv_dzh), d.y);
}

// Transparent ends: what the diagonal of a system's end row loses (edge: the
// field there, inner: beside it), and what the right-hand side of the first
// and last system gains.  Out of line: few rows reach them.
__device__ __noinline__ double2 adi_tbc_diag(double2 edge, double2 inner, double kd2) {
  if (!(hypot(inner.x, inner.y) > 1e-6)) return mk(0.0, 0.0);
  return cx_div_real_rn(tbc_factor(edge, inner), kd2);
}
__device__ __noinline__ double2 adi_tbc_rhs(double2 edge, double2 inner, double kd2) {
  if (!(hypot(inner.x, inner.y) > 1e-6)) return mk(0.0, 0.0);
  return cx_div_real_rn(cx_mul_rn(tbc_factor(edge, inner), edge), kd2);
}

__device__ __forceinline__ double2 crecip_newton(double2 b) {
  const double r = rcp_newton(fma(b.x, b.x, b.y * b.y));
  return mk(b.x * r, -b.y * r);
}

__device__ __forceinline__ double2 shfl_up2(double2 v, int d) {
  return mk(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}
__device__ __forceinline__ double2 shfl_down2(double2 v, int d) {
  return mk(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
}
template <int BYTES>
__device__ __forceinline__ void adi_cp_async(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "n"(BYTES)
               : "memory");
}

// Shared memory of the general half step: G + 2 staged systems, the diagonals
// of its G, and the reduction's buffers for more than one warp a system (in
// the place of the diagonals for the longest systems, whose staging fills
// shared memory).
__host__ __device__ constexpr bool adi_own_red(int M, int W) { return W > 1 && M * W < 36; }
template <typename R, int M, int W, int G> constexpr size_t adi_chunk_smem() {
  return sizeof(typename Cx<R>::T) * (G + 2) * (32 * W * M) + sizeof(double2) * G * (32 * W * M) +
         (adi_own_red(M, W) ? sizeof(double2) * G * 8 * 32 * W : 0);
}

// General half step (planes with material, transparent ends): G systems a
// CTA, W warps a system, thread c of a system owning rows c*M .. c*M+M-1.
//
// With the off-diagonal s on both sides a chunk's rows but the last are
// eliminated in one forward sweep, x_i + cp_i x_(i+1) = y_i + p_i X_(c-1), X_c
// the value of chunk c's last row, p_i the running product of -cp; the same
// sweep accumulates x_0 = Y0 + P0 X_(c-1) + Q0 X_c as Y0 = sum pi_i y_i, P0 =
// sum pi_i p_i, Q0 = p_(M-2) (pi_i = p_(i-1); the matrix is symmetric).  The
// last rows then form a symmetric tridiagonal system with one unknown a
// thread, solved by parallel cyclic reduction -- in registers with shuffles
// for one warp a system, through double-buffered shared memory and a named
// barrier a level for more.  Each thread adds its carry-in and substitutes
// back.  One reciprocal a row and one a reduction level.
//
// What bounds it: the latency of the row chain (reciprocal, then the products
// that wait for it) with few warps an SM, about 10 cycles an instruction and
// warp; FP64 issue is about 56 operations a point (19 % of the pipe at 513
// nodes).  So a system is spread over several warps with short chunks, and
// the diagonals -- the only part that needs the material lookups, divisions
// and branches -- are formed for the whole CTA in staging order before the
// unrolled sweep, while the field's copies arrive.  Inlined into the sweep
// they outgrow the instruction cache (21 against 14 us a half step at 513).
//
// Measured, whole steps of a sphere that fills the domain (FP64, us a step,
// before: chunks of 8 rows, two unknowns a chunk, cyclic reduction over the
// CTA with a barrier a level, systems padded to 8 * 2^k): 150 nodes 43.4 ->
// 11.1, 256: 42.1 -> 12.7, 600: 98 -> 31.6, 700: 101 -> 39.3, 1024: 108 ->
// 56.3, 1500: 407 -> 144; 513 over 64 steps, 20 of them vacuum, 58.4 -> 21.1.
template <typename R, int M, int W, int G, bool TBC>
__global__ void __launch_bounds__(32 * W *G) adi_chunk_kernel(const __grid_constant__ AdiHalf h) {
  using C = typename Cx<R>::T;
  constexpr int P = 32 * W, T = P * G, LD = P * M, RW = G + 2;
  static_assert(M % 2 == 1, "an odd chunk stride: a warp's lanes hit different bank groups");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2 *diag = reinterpret_cast<double2 *>(smem_raw);  // G x LD
  constexpr bool OWN_RED = adi_own_red(M, W);
  C *tile = reinterpret_cast<C *>(diag + G * LD + (OWN_RED ? G * 8 * P : 0));  // RW x LD
  const int n = h.n;
  const int tid = threadIdx.x;
  const int s_base = blockIdx.x * G;
  const C *in = reinterpret_cast<const C *>(h.in);
  C *out = reinterpret_cast<C *>(h.out);
  const bool interleaved = h.stride_sys == 1;
  const int nsys = n - s_base < G ? n - s_base : G;  // the last CTA may hold fewer
  constexpr int PPI = T / RW;  // x half step: positions staged at a time
  constexpr int PPO = T / G;   // and stored

  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  // ---- stage systems s_base-1 .. s_base+G; outside the grid the field is zero
  if (interleaved) {
    // adjacent systems are adjacent in memory: consecutive threads take them
    const int g = tid % RW, sys = s_base - 1 + g;
    if (tid < PPI * RW) {
      C *dst = tile + g * LD;
      if (sys >= 0 && sys < n)
        for (int p = tid / RW; p < n; p += PPI)
          adi_cp_async<sizeof(C)>(dst + p, in + (long long)p * h.stride_pos + sys);
      else
        for (int p = tid / RW; p < n; p += PPI) dst[p] = C{};
    }
  } else {
    for (int g = 0; g < RW; ++g) {
      const int sys = s_base - 1 + g;
      const C *src = in + (long long)sys * h.stride_sys;
      C *dst = tile + g * LD;
      if (sys >= 0 && sys < n)
        for (int p = tid; p < n; p += T) adi_cp_async<sizeof(C)>(dst + p, src + p);
      else
        for (int p = tid; p < n; p += T) dst[p] = C{};
    }
  }
  const double q = __ddiv_rn(0.5, h.kd2_impl);  // the off-diagonal is -i q
  const double inv_impl = __ddiv_rn(1.0, h.kd2_impl);
  const double inv_expl = __ddiv_rn(1.0, h.kd2_expl);
  const double hk = 0.5 * inv_expl;
  // ---- diagonals, while the field arrives
  if (interleaved) {
    const int gg = tid % G, sys = s_base + gg;
    const double y = __dadd_rn(h.ymin, __dmul_rn((double)sys, h.dy));
    if (tid < PPO * G)
      for (int p = tid / G; p < LD; p += PPO) {
        const double x = __dadd_rn(h.xmin, __dmul_rn((double)p, h.dx));
        diag[gg * LD + p] = p < n && gg < nsys ? adi_diag(h, x, y, (long long)p * n + sys, inv_impl)
                                               : mk(kAdiPad, 0.0);
      }
  } else {
#pragma unroll 1
    for (int gg = 0; gg < G; ++gg) {
      const int sys = s_base + gg;
      const double x = __dadd_rn(h.xmin, __dmul_rn((double)sys, h.dx));
      for (int p = tid; p < LD; p += T) {
        const double y = __dadd_rn(h.ymin, __dmul_rn((double)p, h.dy));
        diag[gg * LD + p] = p < n && gg < nsys ? adi_diag(h, x, y, (long long)sys * n + p, inv_impl)
                                               : mk(kAdiPad, 0.0);
      }
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();

  const int g = tid / P, c = tid % P;
  const int s = s_base + g;
  const int p0 = c * M;
  const C *ctr = tile + (g + 1) * LD + p0;
  const C *lft = ctr - LD, *rgt = ctr + LD;
  double2 *dgs = diag + g * LD + p0;
  auto smul = [q](double2 z) { return mk(q * z.y, -q * z.x); };  // off-diagonal * z
  if (TBC && g < nsys) {
    // the diagonal of the system's two end rows
    const C *sysv = tile + (g + 1) * LD;
    if (c == 0) dgs[0] = cx_sub_rn(dgs[0], adi_tbc_diag(to_d(sysv[0]), to_d(sysv[1]), h.kd2_impl));
    if (p0 <= n - 1 && n - 1 < p0 + M)
      dgs[n - 1 - p0] = cx_sub_rn(
          dgs[n - 1 - p0], adi_tbc_diag(to_d(sysv[n - 1]), to_d(sysv[n - 2]), h.kd2_impl));
  }

  // diagonal and right-hand side of row m (position p0 + m) of this chunk
  auto row = [&](int m, double2 &dg, double2 &rh) {
    dg = dgs[m];
    rh = mk(0.0, 0.0);
    if (p0 + m >= n || g >= nsys) return;
    // (1/dz - i/(k d_e^2)) u + 0.5 i (u_left + u_right)/(k d_e^2)
    const double2 r = cmul(mk(h.inv_dzh, -inv_expl), to_d(ctr[m]));
    const double2 nb = cadd(to_d(lft[m]), to_d(rgt[m]));
    rh = mk(fma(-hk, nb.y, r.x), fma(hk, nb.x, r.y));
    if (TBC && (s == 0 || s == n - 1))
      rh = cx_add_rn(rh, adi_tbc_rhs(to_d(ctr[m]), to_d(s == n - 1 ? lft[m] : rgt[m]), h.kd2_expl));
  };

  // ---- forward sweep over rows 0 .. M-2
  double2 cp[M - 1], yv[M - 1];
  double2 pi = mk(1.0, 0.0), y0 = mk(0.0, 0.0), pp0 = mk(0.0, 0.0);
#pragma unroll
  for (int m = 0; m < M - 1; ++m) {
    double2 dg, rh;
    row(m, dg, rh);
    if (m > 0) {
      dg = csub(dg, smul(cp[m - 1]));
      rh = csub(rh, smul(yv[m - 1]));
    }
    const double2 inv = crecip_newton(dg);
    cp[m] = smul(inv);
    yv[m] = cmul(rh, inv);
    y0 = cfma(pi, yv[m], y0);
    const double2 t = cmul(cp[m], pi);
    const double2 pn = mk(-t.x, -t.y);
    pp0 = cfma(pi, pn, pp0);
    pi = pn;
  }
  // ---- the last row's equation a X_(c-1) + b X_c + e X_(c+1) = d
  double2 b, d;
  row(M - 1, b, d);
  b = csub(b, smul(cp[M - 2]));
  d = csub(d, smul(yv[M - 2]));
  double2 a = c > 0 ? smul(pi) : mk(0.0, 0.0);
  double2 e = mk(0.0, 0.0);
  double2 x, xl;
  if constexpr (W == 1) {
    const double2 ry = shfl_down2(y0, 1), rp = shfl_down2(pp0, 1), rq = shfl_down2(pi, 1);
    if (c < P - 1) {
      b = cadd(b, smul(rp));
      d = csub(d, smul(ry));
      e = smul(rq);
    }
#pragma unroll
    for (int sh = 1; sh < P; sh <<= 1) {
      const double2 r = crecip_newton(b);
      const double2 dn = cmul(d, r), an = cmul(a, r), en = cmul(e, r);
      const double2 rl = shfl_up2(r, sh), dl = shfl_up2(dn, sh), al = shfl_up2(an, sh);
      const double2 rr = shfl_down2(r, sh), dr = shfl_down2(dn, sh), er = shfl_down2(en, sh);
      // lanes without a neighbour at this distance hold a = 0 (e = 0)
      b = csub(b, cadd(cmul(a, cmul(a, rl)), cmul(e, cmul(e, rr))));
      d = csub(d, cadd(cmul(a, dl), cmul(e, dr)));
      const double2 a2 = cmul(a, al), e2 = cmul(e, er);
      a = mk(-a2.x, -a2.y);
      e = mk(-e2.x, -e2.y);
    }
    x = cmul(d, crecip_newton(b));
    xl = shfl_up2(x, 1);
  } else {
    // two alternating buffers of P x {reciprocal, d, a, e}: a thread writes
    // a buffer again only after the barrier that follows every read of it
    double2 *buf = OWN_RED ? diag + G * LD + g * 8 * P : diag + g * LD;
    if (!OWN_RED) group_sync(1 + g, P);  // the system's diagonals are read
    buf[c] = y0;
    buf[P + c] = pp0;
    buf[2 * P + c] = pi;
    group_sync(1 + g, P);
    if (c < P - 1) {
      b = cadd(b, smul(buf[P + c + 1]));
      d = csub(d, smul(buf[c + 1]));
      e = smul(buf[2 * P + c + 1]);
    }
    int k = 1;
#pragma unroll 1
    for (int sh = 1; sh < P; sh <<= 1, k ^= 1) {
      double2 *w = buf + k * 4 * P;
      const double2 r = crecip_newton(b);
      w[c] = r;
      w[P + c] = cmul(d, r);
      w[2 * P + c] = cmul(a, r);
      w[3 * P + c] = cmul(e, r);
      group_sync(1 + g, P);
      double2 nb = b, nd = d, na = mk(0.0, 0.0), ne = mk(0.0, 0.0);
      if (c >= sh) {
        const int j = c - sh;
        nb = csub(nb, cmul(a, cmul(a, w[j])));
        nd = csub(nd, cmul(a, w[P + j]));
        na = cmul(a, w[2 * P + j]);
      }
      if (c + sh < P) {
        const int j = c + sh;
        nb = csub(nb, cmul(e, cmul(e, w[j])));
        nd = csub(nd, cmul(e, w[P + j]));
        ne = cmul(e, w[3 * P + j]);
      }
      b = nb;
      d = nd;
      a = mk(-na.x, -na.y);
      e = mk(-ne.x, -ne.y);
    }
    x = cmul(d, crecip_newton(b));
    buf[k * 4 * P + c] = x;
    group_sync(1 + g, P);
    xl = c > 0 ? buf[k * 4 * P + c - 1] : mk(0.0, 0.0);
  }
  // ---- carry-in, then back substitution; results through the tile
  if (c > 0) {
    double2 t = xl;
#pragma unroll
    for (int m = 0; m < M - 1; ++m) {
      t = cmul(cp[m], t);
      t = mk(-t.x, -t.y);
      yv[m] = cadd(yv[m], t);
    }
  }
  __syncthreads();  // every read of the staged systems is done
  C *dst = tile + (g + 1) * LD + p0;
  dst[M - 1] = from_d<R>(x);
#pragma unroll
  for (int m = M - 2; m >= 0; --m) {
    x = csub(yv[m], cmul(cp[m], x));
    dst[m] = from_d<R>(x);
  }
  __syncthreads();
  C *save = reinterpret_cast<C *>(h.save);
  if (interleaved) {
    const int gg = tid % G;
    if (tid < PPO * G && gg < nsys)
      for (int p = tid / G; p < n; p += PPO) {
        const long long off = (long long)p * h.stride_pos + s_base + gg;
        const C v = tile[(gg + 1) * LD + p];
        out[off] = v;
        if (save) save[off] = v;
      }
  } else {
    for (int gg = 0; gg < nsys; ++gg) {
      const long long base = (long long)(s_base + gg) * h.stride_sys;
      for (int p = tid; p < n; p += T) {
        const C v = tile[(gg + 1) * LD + p];
        out[base + p] = v;
        if (save) save[base + p] = v;
      }
    }
  }
}

// Same half step when the matrix is the vacuum one for every system: the
// right-hand side stencil is fused with the two substitution scans of the
// precomputed factorisation (scan_solve.cuh).  No material, no boundary terms.
template <typename R, int N, int M, int G>
__global__ void __launch_bounds__(G *(N / M)) adi_const_kernel(const AdiHalf h,
                                                               const double2 *__restrict__ gtab,
                                                               const double2 *__restrict__ htab) {
  using C = typename Cx<R>::T;
  constexpr int P = N / M;
  constexpr int T = G * P;
  constexpr int ld = N + N / 8 + 2;  // padded row (pad8)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C *tile = reinterpret_cast<C *>(smem_raw);
  double2 *gs = reinterpret_cast<double2 *>(smem_raw + ((sizeof(C) * (G + 2) * ld + 15) & ~size_t(15)));
  double2 *hs = gs + (N + N / 8);
  Affine *scratch = reinterpret_cast<Affine *>(hs + (N + N / 8));
  const int tid = threadIdx.x;
  const int s_base = blockIdx.x * G;
  const C *in = reinterpret_cast<const C *>(h.in);
  C *out = reinterpret_cast<C *>(h.out);
  const bool interleaved = h.stride_sys == 1;
  constexpr int rows = G + 2;
  for (int idx = tid; idx < rows * N; idx += T) {
    int g, p;
    if (interleaved) {
      p = idx / rows;
      g = idx - p * rows;
    } else {
      g = idx / N;
      p = idx - g * N;
    }
    const int s = s_base - 1 + g;
    C v = from_d<R>(mk(0.0, 0.0));
    if (s >= 0 && s < N) v = in[(long long)p * h.stride_pos + (long long)s * h.stride_sys];
    tile[g * ld + pad8(p)] = v;
  }
  for (int i = tid; i < N; i += T) {
    gs[pad8(i)] = gtab[i];
    hs[pad8(i)] = htab[i];
  }
  __syncthreads();
  const int g = tid / P, c = tid - g * P;
  const int s = s_base + g;
  const int p0 = c * M;
  const double inv_kd2_expl = __ddiv_rn(1.0, h.kd2_expl);
  const double hk = 0.5 * inv_kd2_expl;
  const C *ctr = tile + (g + 1) * ld;
  const C *lft = tile + g * ld;
  const C *rgt = tile + (g + 2) * ld;
  double2 r[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int p = p0 + m;
    double2 rr = cmul(mk(h.inv_dzh, -inv_kd2_expl), to_d(ctr[pad8(p)]));
    double2 nb = mk(0.0, 0.0);
    if (s > 0) nb = to_d(lft[pad8(p)]);
    if (s < N - 1) nb = cadd(nb, to_d(rgt[pad8(p)]));
    r[m] = mk(fma(-hk, nb.y, rr.x), fma(hk, nb.x, rr.y));
  }
  const_solve<M, P>(r, gs, hs, p0, scratch);
  __syncthreads();  // every read of the staged tile is done
  C *dst = tile + (g + 1) * ld;
#pragma unroll
  for (int m = 0; m < M; ++m) dst[pad8(p0 + m)] = from_d<R>(r[m]);
  __syncthreads();
  C *save = reinterpret_cast<C *>(h.save);
  for (int idx = tid; idx < G * N; idx += T) {
    int gg, p;
    if (interleaved) {
      p = idx / G;
      gg = idx - p * G;
    } else {
      gg = idx / N;
      p = idx - gg * N;
    }
    const long long off = (long long)p * h.stride_pos + (long long)(s_base + gg) * h.stride_sys;
    const C v = tile[(gg + 1) * ld + pad8(p)];
    out[off] = v;
    if (save) save[off] = v;
  }
}

template <typename R, int N, int G>
static cudaError_t adi_const_launch(const AdiHalf &h, const void *g, const void *hh, cudaStream_t s) {
  using C = typename Cx<R>::T;
  constexpr int M = 8, P = N / M, T = G * P;
  constexpr size_t smem = ((sizeof(C) * (G + 2) * (N + N / 8 + 2) + 15) & ~size_t(15)) +
                          2 * sizeof(double2) * (N + N / 8) + sizeof(Affine) * (T / 32 + 1);
  auto k = adi_const_kernel<R, N, M, G>;
  {
    const cudaError_t attr = raise_dynamic_smem((const void *)k, (int)smem);
    if (attr != cudaSuccess) return attr;
  }
  k<<<N / G, T, smem, s>>>(h, (const double2 *)g, (const double2 *)hh);
  return cudaGetLastError();
}

// Vacuum half step, n <= 1024, one wave: G systems per CTA so that ceil(n / G)
// CTAs fit the 148 SMs at once (G = 7 at n = 1024: 147 CTAs).  The solve is FP64;
// complex64 fields are widened as they are staged and rounded as they leave.
// Systems are solved with N rows, N the smallest of 64, 128, 256, 512, 768
// and 1024 that holds the grid's n (h.n): rows n .. N-1 are decoupled (their
// factors g = 1, h = 0, right-hand sides zero, nothing copied in or out),
// so grids of any size up to 1024 take this path.
// The G + 2 staged rows (G systems and their two stencil halos) arrive by
// coalesced 16-byte cp.async copies, the factor tables (one 64 KB block at
// n = 1024) by one TMA bulk copy counted on an mbarrier; results leave by
// coalesced stores.  (Bulk copies per position run or per chunk -- 32 to 256
// bytes each -- measured slower than per-thread copies: the copy engine's
// per-request cost dominates at these sizes.)
//
// Compute: the CTA's systems form groups of S (two; one where a CTA holds just
// two systems); a thread owns one chunk of M rows of every system of its group.
// Each staged value is read from shared memory once and serves the three
// stencils it enters, each factor-table entry serves all systems of the
// group, and the sweeps run the group's independent recurrences side by
// side.  The chunk-carry scans handle the group's systems together: the
// multiplier product is the same for all of them (one matrix), the carry
// differs per system (multi_exclusive_scan).
//
// Shared-memory layouts keep the per-chunk reads of the solve and the
// copies in memory order free of bank conflicts:
//   XH (x half step, the G + 2 systems of a position adjacent in memory):
//      entry (c, m, g) at c*(M*(G+2) + 1) + m*(G+2) + g, one spare entry after
//      each chunk;
//   YH (y half step, a system is a row): entry (c, m, g) at
//      g*P*(M+1) + c*(M+1) + m, one spare entry after each chunk.
// The tables [g | h | pf | pb] (Thomas factors and the in-chunk products of
// the multipliers) are host-built in chunk-transposed slots
// (adi_const_staged_tables) and copied in as one block.  The same tile holds
// the results (row g + 1 of system g) for the stores.
template <int N, int M, int G, bool XH>
struct AdiWaveTile {
  static constexpr int P = N / M, RW = G + 2;
  static constexpr int SIZE = XH ? N * RW + P : RW * P * (M + 1);
  __device__ static __forceinline__ int at(int c, int m, int g) {
    return XH ? c * (M * RW + 1) + m * RW + g : g * P * (M + 1) + c * (M + 1) + m;
  }
};

__device__ __forceinline__ void adi_cp_async16(void *smem, const void *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(smem)), "l"(gmem) : "memory");
}


template <bool DOWN>
__device__ __forceinline__ double2 shfl2(double2 v, int d) {
  if (DOWN) return mk(__shfl_down_sync(0xffffffffu, v.x, d), __shfl_down_sync(0xffffffffu, v.y, d));
  return mk(__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d));
}

// Exclusive scan of chunk transfers y_out = a*y_in + b[j] over the P threads
// of a group (P a multiple of 32, the group starting at a warp boundary),
// S systems at once with a common multiplier a.  REV scans in decreasing
// chunk order.  On return (a, b) hold the composition of the transfers of
// the chunks before this one in scan order (identity for the first).
// scratch: (S + 1) * P / 32 entries for this group; bar: its named barrier.
template <int P, int S, bool REV>
__device__ __forceinline__ void multi_exclusive_scan(double2 &a, double2 (&b)[S], double2 *scratch,
                                                     int gtid, int bar) {
  const int lane = threadIdx.x & 31;
  double2 ia = a, ib[S];
#pragma unroll
  for (int j = 0; j < S; ++j) ib[j] = b[j];
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const double2 oa = shfl2<REV>(ia, d);
    double2 ob[S];
#pragma unroll
    for (int j = 0; j < S; ++j) ob[j] = shfl2<REV>(ib[j], d);
    if (REV ? lane + d < 32 : lane >= d) {
#pragma unroll
      for (int j = 0; j < S; ++j) ib[j] = cfma(ia, ob[j], ib[j]);
      ia = cmul(ia, oa);
    }
  }
  double2 ea = shfl2<REV>(ia, 1), eb[S];
#pragma unroll
  for (int j = 0; j < S; ++j) eb[j] = shfl2<REV>(ib[j], 1);
  if (REV ? lane == 31 : lane == 0) {
    ea = mk(1.0, 0.0);
#pragma unroll
    for (int j = 0; j < S; ++j) eb[j] = mk(0.0, 0.0);
  }
  if constexpr (P > 32) {
    constexpr int W = P / 32;
    const int w = gtid >> 5;
    group_sync(bar, P);  // the previous scan's readers are done with scratch
    if (lane == (REV ? 0 : 31)) {
      scratch[w * (S + 1)] = ia;
#pragma unroll
      for (int j = 0; j < S; ++j) scratch[w * (S + 1) + 1 + j] = ib[j];
    }
    group_sync(bar, P);
    double2 pa = mk(1.0, 0.0), pb[S];
#pragma unroll
    for (int j = 0; j < S; ++j) pb[j] = mk(0.0, 0.0);
#pragma unroll
    for (int k = 1; k < W; ++k) {
      const int v = REV ? W - k : k - 1;  // warps before this one in scan order
      if (REV ? v > w : v < w) {
        const double2 ta = scratch[v * (S + 1)];
#pragma unroll
        for (int j = 0; j < S; ++j) pb[j] = cfma(ta, pb[j], scratch[v * (S + 1) + 1 + j]);
        pa = cmul(ta, pa);
      }
    }
    // compose(pre, ex): apply the preceding warps, then this warp's lanes
#pragma unroll
    for (int j = 0; j < S; ++j) eb[j] = cfma(ea, pb[j], eb[j]);
    ea = cmul(ea, pa);
  }
  a = ea;
#pragma unroll
  for (int j = 0; j < S; ++j) b[j] = eb[j];
}

// Right-hand sides and solve of systems sys0 .. sys0+SC-1 of this CTA for
// chunk c: r[j][m] holds the solution of row c*M + m of system sys0 + j.
template <int N, int M, int G, bool XH, int SCAP, int S>
__device__ __forceinline__ void adi_group_solve(double2 (&r)[SCAP][M], const AdiHalf &h,
                                                const double2 *tile, const double2 *gs,
                                                const double2 *hs, const double2 *pf,
                                                const double2 *pb, double2 *scratch, int sys0,
                                                int s_base, int c, int gtid, int bar) {
  using L = AdiWaveTile<N, M, G, XH>;
  constexpr int P = N / M;
  const double inv_kd2_expl = __ddiv_rn(1.0, h.kd2_expl);
  const double hk = 0.5 * inv_kd2_expl;
  const double2 coef = mk(h.inv_dzh, -inv_kd2_expl);
  // table chunk: inside the run of identical chunks every thread reads the
  // run's first chunk, so a warp's table reads there are broadcasts
  const int ct = (c > h.tab_c0 && c < h.tab_c1) ? h.tab_c0 : c;
#pragma unroll
  for (int m = 0; m < M; ++m) {
    double2 v[S + 2];
#pragma unroll
    for (int k = 0; k < S + 2; ++k) v[k] = tile[L::at(c, m, sys0 + k)];
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const int s = s_base + sys0 + j;  // s >= h.n: padding system, all zero
      const double2 rr = cmul(coef, v[j + 1]);
      double2 nb = mk(0.0, 0.0);
      if (s > 0) nb = v[j];
      if (s < h.n - 1) nb = cadd(nb, v[j + 2]);
      r[j][m] = mk(fma(-hk, nb.y, rr.x), fma(hk, nb.x, rr.y));
    }
  }
  // forward, zero carry-in: y_i = g_i r_i + h_i y_{i-1}
  double2 y[S];
  {
    const double2 g0 = gs[cslot<M, P>(ct, 0)];
#pragma unroll
    for (int j = 0; j < S; ++j) r[j][0] = y[j] = cmul(g0, r[j][0]);
  }
#pragma unroll
  for (int m = 1; m < M; ++m) {
    const int k = cslot<M, P>(ct, m);
    const double2 gm = gs[k], hm = hs[k];
#pragma unroll
    for (int j = 0; j < S; ++j) r[j][m] = y[j] = cfma(hm, y[j], cmul(gm, r[j][m]));
  }
  double2 a = pf[cslot<M, P>(ct, M - 1)];
  multi_exclusive_scan<P, S, false>(a, y, scratch, gtid, bar);
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const double2 f = pf[cslot<M, P>(ct, m)];
#pragma unroll
    for (int j = 0; j < S; ++j) r[j][m] = cfma(f, y[j], r[j][m]);
  }
  // backward, zero carry-in: x_i = y_i + h_i x_{i+1}
  double2 x[S];
#pragma unroll
  for (int j = 0; j < S; ++j) x[j] = r[j][M - 1];
#pragma unroll
  for (int m = M - 2; m >= 0; --m) {
    const double2 hm = hs[cslot<M, P>(ct, m)];
#pragma unroll
    for (int j = 0; j < S; ++j) r[j][m] = x[j] = cfma(hm, x[j], r[j][m]);
  }
  a = pb[cslot<M, P>(ct, 0)];
  multi_exclusive_scan<P, S, true>(a, x, scratch, gtid, bar);
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const double2 f = pb[cslot<M, P>(ct, m)];
#pragma unroll
    for (int j = 0; j < S; ++j) r[j][m] = cfma(f, x[j], r[j][m]);
  }
}

// Systems per group S: a thread owns one chunk of M rows of the S systems of
// its group; NG = ceil(G / S) groups of P = n/M threads each (the last group
// may hold fewer systems).
// Complex64 fields are widened as they are staged and rounded as they leave.
template <typename R, int N, int M, int G, int S, bool XH>
__global__ void __launch_bounds__(((G + S - 1) / S) * (N / M), 1)
    adi_const_wave_kernel(const AdiHalf h, const double2 *__restrict__ tabs) {
  using L = AdiWaveTile<N, M, G, XH>;
  constexpr int P = N / M;
  constexpr int NG = (G + S - 1) / S;
  constexpr int T = NG * P;
  constexpr int RW = G + 2;
  constexpr int SL = G - (NG - 1) * S;  // systems of the last group
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw);
  double2 *gs = reinterpret_cast<double2 *>(smem_raw + 16);
  double2 *hs = gs + N;
  double2 *pf = hs + N;
  double2 *pb = pf + N;
  double2 *scratch = pb + N;  // (S + 1) * P / 32 per group
  double2 *tile = scratch + NG * (S + 1) * (P / 32);
  __shared__ int staged_ok;
  const int tid = threadIdx.x;
  const int group = tid / P, gtid = tid % P;
  const int s_base = blockIdx.x * G;
  using C = typename Cx<R>::T;
  const C *in = reinterpret_cast<const C *>(h.in);
  C *out = reinterpret_cast<C *>(h.out);
  auto stage = [](double2 *dst, const C *src) {
    if constexpr (sizeof(R) == 8) adi_cp_async16(dst, src);
    else *dst = to_d(*src);
  };
  const int nr = h.n;  // systems, and positions per system (N: rows solved)
  // staged systems s_base - 1 + g exist for g in [g_lo, g_hi)
  const int g_lo = s_base == 0 ? 1 : 0;
  const int g_hi = nr - s_base + 1 < RW ? nr - s_base + 1 : RW;
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_arrive_expect_tx(bar, (unsigned)(sizeof(double2) * 4 * N));
  }
  // staged rows outside the grid (first and last CTA) and the padding
  // positions nr .. N-1 are zero
  for (int g = 0; g < RW; ++g)
    for (int p = (g < g_lo || g >= g_hi) ? tid : nr + tid; p < N; p += T)
      tile[L::at(p / M, p % M, g)] = mk(0.0, 0.0);
  __syncthreads();
  if (tid == 0) bulk_load(gs, tabs, (unsigned)(sizeof(double2) * 4 * N), bar);
  // Programmatic dependent launch: everything above (barrier set-up, zero
  // rows, the table copy) does not depend on the previous kernel in the
  // stream, so it may overlap that kernel's tail; the field is read and
  // written only after the previous grid has completed and its writes are
  // visible.  The next kernel may likewise start its own set-up early.
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if constexpr (XH) {
    // the RW staged systems of a position are adjacent in memory:
    // consecutive threads take consecutive systems
    constexpr int PPI = T / RW;  // positions per pass
    const int g = tid % RW;
    if (tid < PPI * RW && g >= g_lo && g < g_hi) {
      const C *src = in + (s_base - 1 + g);
      for (int p = tid / RW; p < nr; p += PPI)
        stage(tile + L::at(p / M, p % M, g), src + (long long)p * h.stride_pos);
    }
  } else {
#pragma unroll 1
    for (int g = g_lo; g < g_hi; ++g) {
      const C *src = in + (long long)(s_base - 1 + g) * h.stride_sys;
      for (int p = tid; p < nr; p += T) stage(tile + L::at(p / M, p % M, g), src + p);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  if (tid == 0) {
    const bool ok = mbar_wait_bounded(bar, 0, 2000000000ull);
    if (!ok) {
      atomicAdd(h.timeouts, 1u);
      mbar_wait_bounded(bar, 0, 2000000000ull);  // the table copy may still be in flight
    }
    staged_ok = ok;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  if (!staged_ok) return;
  (void)mbar_try_wait(bar, 0);  // completed phase: orders the copied tables for this thread
  double2 r[S][M];
  double2 *gscr = scratch + group * (S + 1) * (P / 32);
  if (SL == S || group < NG - 1)
    adi_group_solve<N, M, G, XH, S, S>(r, h, tile, gs, hs, pf, pb, gscr, group * S, s_base, gtid,
                                       gtid, 1 + group);
  else
    adi_group_solve<N, M, G, XH, S, SL>(r, h, tile, gs, hs, pf, pb, gscr, group * S, s_base, gtid,
                                        gtid, 1 + group);
  __syncthreads();  // every read of the staged tile is done
  const int ns = group < NG - 1 ? S : SL;
#pragma unroll
  for (int j = 0; j < S; ++j)
    if (j < ns) {
#pragma unroll
      for (int m = 0; m < M; ++m) tile[L::at(gtid, m, group * S + j + 1)] = r[j][m];
    }
  __syncthreads();
  C *save = reinterpret_cast<C *>(h.save);
  const int nsys = nr - s_base < G ? nr - s_base : G;  // the last CTA may hold fewer
  if constexpr (XH) {
    // consecutive threads write consecutive systems of a position
    constexpr int PPI = T / G;
    const int gg = tid % G;
    if (tid < PPI * G && gg < nsys) {
      for (int p = tid / G; p < nr; p += PPI) {
        const C v = from_d<R>(tile[L::at(p / M, p % M, gg + 1)]);
        const long long off = (long long)p * h.stride_pos + s_base + gg;
        out[off] = v;
        if (save) save[off] = v;
      }
    }
  } else {
#pragma unroll 1
    for (int gg = 0; gg < nsys; ++gg) {
      const long long base = (long long)(s_base + gg) * h.stride_sys;
      for (int p = tid; p < nr; p += T) {
        const C v = from_d<R>(tile[L::at(p / M, p % M, gg + 1)]);
        out[base + p] = v;
        if (save) save[base + p] = v;
      }
    }
  }
}

// cp.async completion counted on an mbarrier: when every cp.async this
// thread issued before the instruction has landed, the barrier sees one
// arrival (noinc: the arrival is one of the count the barrier was set up
// with).
__device__ __forceinline__ void cp_async_mbar_arrive(uint64_t *bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(bar))
               : "memory");
}

// Bytes before the factor tables in the one-wave kernels' shared memory: the
// mbarriers (one for the tables and, in the pipelined kernel, one per
// system group), rounded up to 16 bytes.
template <int NG> constexpr size_t adi_wave_bar_bytes() { return 16 * ((NG + 2) / 2 + 1); }

// The one-wave vacuum half step with its staging pipelined against the
// solves.  The staged rows are copied in stages, one per system group in
// group order (stage 0: the rows group 0 reads; stage k: the rows group k
// needs that no earlier stage brought); every thread issues its share of a
// stage's copies and then an asynchronous arrival on that stage's mbarrier,
// so a stage completes when all of its copies (and every earlier stage's)
// have landed.  Each group waits for its own stage and the factor tables
// (its leader with the bounded wait, then the group's named barrier),
// solves, and stores its systems straight from registers: group 0 computes
// while later rows are still arriving, and one group's stores overlap the
// others' solves.  Same arithmetic as adi_const_wave_kernel.
template <int N, int M, int G, int S, bool XH>
__global__ void __launch_bounds__(((G + S - 1) / S) * (N / M), 1)
    adi_pipe_wave_kernel(const AdiHalf h, const double2 *__restrict__ tabs) {
  using L = AdiWaveTile<N, M, G, XH>;
  constexpr int P = N / M;
  constexpr int NG = (G + S - 1) / S;
  constexpr int T = NG * P;
  constexpr int RW = G + 2;
  constexpr int SL = G - (NG - 1) * S;  // systems of the last group
  extern __shared__ __align__(16) unsigned char smem_raw[];
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem_raw);  // [0]: tables, [1 + k]: stage k
  double2 *gs = reinterpret_cast<double2 *>(smem_raw + adi_wave_bar_bytes<NG>());
  double2 *hs = gs + N;
  double2 *pf = hs + N;
  double2 *pb = pf + N;
  double2 *scratch = pb + N;  // (S + 1) * P / 32 per group
  double2 *tile = scratch + NG * (S + 1) * (P / 32);
  __shared__ int group_ok[NG];
  const int tid = threadIdx.x;
  const int group = tid / P, gtid = tid % P;
  const int s_base = blockIdx.x * G;
  const double2 *in = reinterpret_cast<const double2 *>(h.in);
  double2 *out = reinterpret_cast<double2 *>(h.out);
  double2 *save = reinterpret_cast<double2 *>(h.save);
  const int nr = h.n;  // systems, and positions per system (N: rows solved)
  const int g_lo = s_base == 0 ? 1 : 0;
  const int g_hi = nr - s_base + 1 < RW ? nr - s_base + 1 : RW;
  if (tid == 0) {
    mbar_init(bar, 1);
    for (int k = 0; k < NG; ++k) mbar_init(bar + 1 + k, T);
    mbar_arrive_expect_tx(bar, (unsigned)(sizeof(double2) * 4 * N));
  }
  // rows outside the grid and the padding positions nr .. N-1 are zero
  for (int g = 0; g < RW; ++g)
    for (int p = (g < g_lo || g >= g_hi) ? tid : nr + tid; p < N; p += T)
      tile[L::at(p / M, p % M, g)] = mk(0.0, 0.0);
  __syncthreads();
  if (tid == 0) bulk_load(gs, tabs, (unsigned)(sizeof(double2) * 4 * N), bar);
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  // stage k brings staged rows [lo_k, hi_k); group k reads rows k*S .. k*S + S + 1
#pragma unroll 1
  for (int k = 0; k < NG; ++k) {
    const int lo = k == 0 ? 0 : k * S + 2;
    const int hi = k == NG - 1 ? RW : (k + 1) * S + 2;
    const int rows = hi - lo;
    if constexpr (XH) {
      // the rows of a position are adjacent in memory: consecutive threads
      // take consecutive rows, then the next position
      for (int i = tid; i < nr * rows; i += T) {
        const int p = i / rows, g = lo + i % rows;
        if (g >= g_lo && g < g_hi)
          adi_cp_async16(tile + L::at(p / M, p % M, g),
                         in + (long long)p * h.stride_pos + (s_base - 1 + g));
      }
    } else {
      for (int g = lo; g < hi; ++g) {
        if (g < g_lo || g >= g_hi) continue;
        const double2 *src = in + (long long)(s_base - 1 + g) * h.stride_sys;
        for (int p = tid; p < nr; p += T) adi_cp_async16(tile + L::at(p / M, p % M, g), src + p);
      }
    }
    cp_async_mbar_arrive(bar + 1 + k);
  }
  // this group's rows and the tables
  if (gtid == 0) {
    bool ok = mbar_wait_bounded(bar + 1 + group, 0, 2000000000ull);
    ok = mbar_wait_bounded(bar, 0, 2000000000ull) && ok;
    if (!ok) atomicAdd(h.timeouts, 1u);
    group_ok[group] = ok;
  }
  group_sync(1 + group, P);
  // a group whose wait ran out skips its solve but still reaches the CTA
  // barriers below (every thread of the CTA passes every barrier); the CTA
  // then leaves without storing
  const bool my_ok = group_ok[group] != 0;
  double2 r[S][M];
  if (my_ok) {
    (void)mbar_try_wait(bar + 1 + group, 0);  // completed phases: order the rows and tables
    (void)mbar_try_wait(bar, 0);
    double2 *gscr = scratch + group * (S + 1) * (P / 32);
    if (SL == S || group < NG - 1)
      adi_group_solve<N, M, G, XH, S, S>(r, h, tile, gs, hs, pf, pb, gscr, group * S, s_base,
                                         gtid, gtid, 1 + group);
    else
      adi_group_solve<N, M, G, XH, S, SL>(r, h, tile, gs, hs, pf, pb, gscr, group * S, s_base,
                                          gtid, gtid, 1 + group);
  }
  // results through the tile to coalesced stores, as in the unpipelined
  // kernel: after every group's reads of the staged rows (one CTA barrier:
  // group 0 waits here for the last group's right-hand sides, while its own
  // solve has already overlapped the later stages' copies), each group
  // writes its systems' rows, and consecutive threads then store
  // consecutive addresses.  (Stores straight from the registers -- each
  // thread's rows strided by the system length -- measured slower than the
  // unpipelined kernel.)
  __syncthreads();  // every group's flag is set and every staged row read
  bool all_ok = true;
#pragma unroll
  for (int k = 0; k < NG; ++k) all_ok = all_ok && group_ok[k] != 0;
  if (!all_ok) {  // the same decision in every thread: nothing writes the flags now
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    return;
  }
  const int ns = group < NG - 1 ? S : SL;
#pragma unroll
  for (int j = 0; j < S; ++j)
    if (j < ns) {
#pragma unroll
      for (int m = 0; m < M; ++m) tile[L::at(gtid, m, group * S + j + 1)] = r[j][m];
    }
  __syncthreads();
  const int nsys = nr - s_base < G ? nr - s_base : G;  // the last CTA may hold fewer
  if constexpr (XH) {
    constexpr int PPI = T / G;
    const int gg = tid % G;
    if (tid < PPI * G && gg < nsys) {
      for (int p = tid / G; p < nr; p += PPI) {
        const double2 v = tile[L::at(p / M, p % M, gg + 1)];
        const long long off = (long long)p * h.stride_pos + s_base + gg;
        out[off] = v;
        if (save) save[off] = v;
      }
    }
  } else {
#pragma unroll 1
    for (int gg = 0; gg < nsys; ++gg) {
      const long long base = (long long)(s_base + gg) * h.stride_sys;
      for (int p = tid; p < nr; p += T) {
        const double2 v = tile[L::at(p / M, p % M, gg + 1)];
        out[base + p] = v;
        if (save) save[base + p] = v;
      }
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");  // copies this thread issued for later groups
}

// The unpipelined one-wave kernel by default; PXP_ADI_PIPE=1 selects the
// pipelined one (measured slower with its stores straight from registers:
// 30.4 against 23.2 us per 1024^2 step).
static bool adi_pipe_enabled() {
  static const bool on = [] {
    const char *e = std::getenv("PXP_ADI_PIPE");
    return e && e[0] == '1';
  }();
  return on;
}

template <typename R, int N, int M, int G, int S, bool XH>
static cudaError_t adi_const_wave_launch_x(const AdiHalf &h, const void *tabs, cudaStream_t s) {
  constexpr int P = N / M, NG = (G + S - 1) / S, T = NG * P;
  constexpr size_t smem = adi_wave_bar_bytes<NG>() +
                          sizeof(double2) * (4 * N + NG * (S + 1) * (P / 32)) +
                          sizeof(double2) * AdiWaveTile<N, M, G, XH>::SIZE;
  static_assert(smem + 16 <= 227 * 1024, "staged ADI tile exceeds shared memory");
  static_assert(P % 32 == 0, "whole warps per group");
  static_assert(NG <= 15, "one named barrier per group");
  auto k = adi_const_wave_kernel<R, N, M, G, S, XH>;
  if constexpr (sizeof(R) == 8)
    if (adi_pipe_enabled()) k = adi_pipe_wave_kernel<N, M, G, S, XH>;
  {
    cudaError_t attr = raise_dynamic_smem((const void *)k, (int)smem);
    // room for one CTA an SM: in a larger carve-out, left behind by a kernel
    // that wanted it (the general half step's), the next half step's CTAs start
    // two to an SM beside this one's and leave other SMs idle (512 nodes after
    // a plane with material: 10.7 -> 13.7 us a step)
    if (attr == cudaSuccess) attr = prefer_smem_carveout((const void *)k, (int)smem, 1);
    if (attr != cudaSuccess) return attr;
  }
  // launched as a programmatic dependent of the previous kernel in the
  // stream (the kernel waits for it with griddepcontrol.wait)
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((h.n + G - 1) / G);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, h, (const double2 *)tabs);
}

template <typename R, int N, int M, int G, int S>
static cudaError_t adi_const_wave_launch(const AdiHalf &h, const void *tabs, cudaStream_t s) {
  if (tabs == nullptr) return cudaErrorInvalidValue;
  return h.stride_sys == 1 ? adi_const_wave_launch_x<R, N, M, G, S, true>(h, tabs, s)
                           : adi_const_wave_launch_x<R, N, M, G, S, false>(h, tabs, s);
}

// Rows a thread of the one-wave kernel for a system length adi_wave_n gives
// (whole warps a system: n / M a multiple of 32), 0 for others.
static int adi_wave_rows(int n) {
  switch (n) {
    case 64: return 2;
    case 128: return 4;
    case 256: case 512: case 768: case 1024: return 8;
    default: return 0;
  }
}

int adi_wave_n(int n) {
  static const int sizes[] = {64, 128, 256, 512, 768, 1024};
  if (n < 4) return 0;
  for (int w : sizes)
    if (n <= w) return w;
  return 0;
}

bool adi_const_staged_tables(int n, const double *g, const double *h, double *out, int run[2]) {
  const int M = adi_wave_rows(n);
  if (M == 0) return false;
  const int P = n / M;
  auto slot = [&](int c, int m) { return m * P + (c ^ (m & 7)); };
  // the device's cmul: (fma(ax, bx, -ay*by), fma(ax, by, ay*bx))
  auto cmul_h = [](const double *a, const double *b, double *o) {
    const double re = std::fma(a[0], b[0], -(a[1] * b[1]));
    const double im = std::fma(a[0], b[1], a[1] * b[0]);
    o[0] = re;
    o[1] = im;
  };
  double *gs = out, *hs = out + 2 * n, *pf = out + 4 * n, *pb = out + 6 * n;
  for (int c = 0; c < P; ++c) {
    double prod[2] = {1.0, 0.0};
    for (int m = 0; m < M; ++m) {
      const int p = c * M + m, k = slot(c, m);
      gs[2 * k] = g[2 * p];
      gs[2 * k + 1] = g[2 * p + 1];
      hs[2 * k] = h[2 * p];
      hs[2 * k + 1] = h[2 * p + 1];
      cmul_h(h + 2 * p, prod, prod);
      pf[2 * k] = prod[0];
      pf[2 * k + 1] = prod[1];
    }
    prod[0] = 1.0;
    prod[1] = 0.0;
    for (int m = M - 1; m >= 0; --m) {
      const int p = c * M + m, k = slot(c, m);
      cmul_h(h + 2 * p, prod, prod);
      pb[2 * k] = prod[0];
      pb[2 * k + 1] = prod[1];
    }
  }
  // Thomas factors of a constant-coefficient matrix reach their limit to the
  // last bit after a few dozen rows, so most chunks' entries coincide
  auto same_chunk = [&](int c0, int c1) {
    for (int t = 0; t < 4; ++t)
      for (int m = 0; m < M; ++m) {
        const double *e0 = out + 2 * ((size_t)t * n + slot(c0, m));
        const double *e1 = out + 2 * ((size_t)t * n + slot(c1, m));
        if (std::memcmp(e0, e1, 2 * sizeof(double)) != 0) return false;
      }
    return true;
  };
  run[0] = run[1] = 0;
  for (int c = 0; c < P;) {
    int e = c + 1;
    while (e < P && same_chunk(c, e)) ++e;
    if (e - c > run[1] - run[0]) {
      run[0] = c;
      run[1] = e;
    }
    c = e;
  }
  if (run[1] - run[0] < 2) run[0] = run[1] = 0;
  return true;
}

// Self-test of the bounded-wait failure path: one thread arms an mbarrier
// for a 16-byte transaction that no copy ever delivers and waits on it with
// the kernels' bounded wait (mbar_wait_bounded) and the given limit.  The
// wait runs out, the kernel records it in the same counter the propagation
// kernels use, and returns; nothing faults and the context stays usable.
__global__ void wait_selftest_kernel(unsigned long long limit_ns, unsigned *timeouts) {
  __shared__ __align__(8) uint64_t bar;
  mbar_init(&bar, 1);
  mbar_arrive_expect_tx(&bar, 16u);
  if (!mbar_wait_bounded(&bar, 0, limit_ns)) atomicAdd(timeouts, 1u);
}

cudaError_t launch_wait_selftest(unsigned long long limit_ns, unsigned *timeouts, cudaStream_t s) {
  wait_selftest_kernel<<<1, 1, 0, s>>>(limit_ns, timeouts);
  return cudaGetLastError();
}

template <typename R>
static cudaError_t adi_half_const(const AdiHalf &h, const void *g, const void *hh,
                                  const void *staged, cudaStream_t s) {
  switch (adi_wave_n(h.n)) {
    case 64: return adi_const_wave_launch<R, 64, 2, 4, 2>(h, staged, s);
    case 128: return adi_const_wave_launch<R, 128, 4, 2, 1>(h, staged, s);
    case 256: return adi_const_wave_launch<R, 256, 8, 2, 1>(h, staged, s);
    // systems a CTA: as few as still make one wave of the 148 SMs (us a step:
    // 290 nodes 9.7 with four, 7.2 with two; 513 16.0 with six, 12.9 with
    // four; 800 23.0 with seven, 19.2 with six); three at 297 .. 444 nodes,
    // a full group of two and a half empty one, are slower than four (440:
    // 12.1 against 11.2)
    case 512:
      if (h.n <= 296) return adi_const_wave_launch<R, 512, 8, 2, 1>(h, staged, s);
      return adi_const_wave_launch<R, 512, 8, 4, 2>(h, staged, s);
    case 768:
      if (h.n <= 592) return adi_const_wave_launch<R, 768, 8, 4, 2>(h, staged, s);
      if (h.n <= 740) return adi_const_wave_launch<R, 768, 8, 5, 2>(h, staged, s);
      return adi_const_wave_launch<R, 768, 8, 6, 2>(h, staged, s);
    case 1024:
      if (h.n <= 888) return adi_const_wave_launch<R, 1024, 8, 6, 2>(h, staged, s);
      return adi_const_wave_launch<R, 1024, 8, 7, 2>(h, staged, s);
    default: break;
  }
  return h.n == 2048 ? adi_const_launch<R, 2048, 2>(h, g, hh, s) : cudaErrorInvalidValue;
}

cudaError_t launch_adi_half_const(Precision p, const AdiHalf &h, const void *g, const void *hh,
                                  const void *staged, cudaStream_t s) {
  return p == kFP64 ? adi_half_const<double>(h, g, hh, staged, s)
                    : adi_half_const<float>(h, g, hh, staged, s);
}

template <typename R, int M, int W, int G>
static cudaError_t adi_chunk_launch_t(const AdiHalf &h, cudaStream_t s) {
  constexpr size_t smem = adi_chunk_smem<R, M, W, G>();
  static_assert(smem <= 227 * 1024, "staged systems exceed shared memory");
  static_assert(W == 1 || G <= 15, "one named barrier per system");
  auto k = h.use_tbc ? adi_chunk_kernel<R, M, W, G, true> : adi_chunk_kernel<R, M, W, G, false>;
  const cudaError_t attr = raise_dynamic_smem((const void *)k, (int)smem);
  if (attr != cudaSuccess) return attr;
  // a programmatic dependent of the previous kernel in the stream: its CTAs
  // start while that kernel drains and wait for it with griddepcontrol.wait
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((h.n + G - 1) / G);
  cfg.blockDim = dim3(32 * W * G);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute la[1];
  la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  la[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = la;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, h);
}

bool adi_size_supported(int n) { return n >= 4 && n <= 2048; }

bool adi_const_supported(int n) { return adi_wave_n(n) > 0 || n == 2048; }

// Rows a thread, warps a system and systems a CTA per grid size.  Two CTAs an
// SM beat one larger CTA (513: G = 2 21.1 us a step, G = 4 22.8) except where
// G = 3 still gives at most one CTA an SM (400: 17.1 against 19.2 with G = 2);
// above 148 CTAs G = 3 leaves SMs with one and SMs with two (513: 31).
// Complex64 tiles are half as large, and fewer, larger CTAs win (513: G = 4
// 22.6, G = 2 27.8; 1024: 17 rows and 2 warps 59.9, 9 rows and 4 warps 64.7).
template <typename R>
static cudaError_t adi_chunk_launch(const AdiHalf &h, cudaStream_t s) {
  const int n = h.n;
  constexpr bool F = sizeof(R) == 4;
  if (n <= 192) return adi_chunk_launch_t<R, 3, 2, 1>(h, s);
  if (n <= 384) return adi_chunk_launch_t<R, 3, 4, 2>(h, s);
  if (n <= 444) return adi_chunk_launch_t<R, 5, 4, 3>(h, s);
  if (n <= 640) return adi_chunk_launch_t<R, 5, 4, F ? 4 : 2>(h, s);
  if (n <= 832) return adi_chunk_launch_t<R, 13, 2, F ? 4 : 2>(h, s);
  if (n <= 1088) {
    if constexpr (F) return adi_chunk_launch_t<R, 17, 2, 4>(h, s);
    else return adi_chunk_launch_t<R, 9, 4, 2>(h, s);
  }
  if (n <= 1664) return adi_chunk_launch_t<R, 13, 4, 2>(h, s);
  return adi_chunk_launch_t<R, 17, 4, 1>(h, s);
}

cudaError_t launch_adi_half(Precision p, const AdiHalf &h, cudaStream_t s) {
  if (!adi_size_supported(h.n)) return cudaErrorInvalidValue;
  return p == kFP64 ? adi_chunk_launch<double>(h, s) : adi_chunk_launch<float>(h, s);
}

}  // namespace pxp
