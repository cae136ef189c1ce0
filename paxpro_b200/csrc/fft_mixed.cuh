// fft_mixed.cuh -- complex FFT of a length whose prime factors are at most 31,
// held in shared memory, shared by the FFTSolver2D kernel (fft1d_mixed.cu) and
// the FFTSolver3D line passes (fft3d_mixed.cu).
//
// Stockham autosort passes over two buffers, one pass a radix: odd radices
// first (their first-pass writes, stride R elements, then hit different bank
// groups), 8 / 4 / 2 last.  A thread takes whole butterflies (or a share of
// one, see pass): R inputs at stride n / R into registers, twiddles, an
// R-point DFT, R outputs at stride NS.  For an odd prime R the inputs are
// folded into sums and differences of the pairs (j, R - j), and each pair of
// outputs (k, R - k) is one chain of real factors, cos on the sums and sin on
// the differences: (R - 1)^2 real multiply-adds a butterfly, about R a point,
// against some 370 operations a point at 513 = 19 * 27 for the chirp-z
// identity that lengths with a larger prime use (two transforms of a
// power-of-two length of at least 2n - 1).  At 31 * 31 = 961 points, its
// worst case, the mixed-radix step still takes 9.7 against 12.2 us.
//
// Only the forward transform exists: the inverse one is the forward one of
// the swapped (im, re) values, swapped back, which the pointwise loops
// between the transforms do as they read and write.
//
// Twiddles come from a table in pass order: the pass with sub-transform
// length NS and radix R holds exp(-2 pi i r k / (NS R)) at offset + (r - 1) *
// NS + k (r = 1 .. R - 1, k < NS), n - 1 entries in all, then the (cos, sin)
// factors of the primes from 11 on (plan.rot); complex128 for FP64 data, split complex64 pairs for complex64 data, whose real constants are
// split too (fft_smem.cuh).
#pragma once
#include <type_traits>

#include "fft_smem.cuh"
#include "pxp_kernels.h"

namespace pxp {
namespace mixed {

// cos and sin of 2 pi m / R, m = 1 .. (R - 1) / 2, for the radices whose
// butterflies are unrolled.
template <int R> struct Rot;
template <> struct Rot<3> {
  static constexpr double c[] = {
      -0.50000000000000000000};
  static constexpr double s[] = {
      0.86602540378443864676};
};
template <> struct Rot<5> {
  static constexpr double c[] = {
      0.30901699437494742410, -0.80901699437494742410};
  static constexpr double s[] = {
      0.95105651629515357212, 0.58778525229247312917};
};
template <> struct Rot<7> {
  static constexpr double c[] = {
      0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
  static constexpr double s[] = {
      0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
};
template <> struct Rot<9> {
  static constexpr double c[] = {
      0.76604444311897803520, 0.17364817766693034885, -0.50000000000000000000,
      -0.93969262078590838405};
  static constexpr double s[] = {
      0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676,
      0.34202014332566873304};
};
template <> struct Rot<11> {
  static constexpr double c[] = {
      0.84125353283118116886, 0.41541501300188642553, -0.14231483827328514044,
      -0.65486073394528506406, -0.95949297361449738989};
  static constexpr double s[] = {
      0.54064081745559758211, 0.90963199535451837141, 0.98982144188093273238,
      0.75574957435425828377, 0.28173255684142969771};
};
template <> struct Rot<13> {
  static constexpr double c[] = {
      0.88545602565320989590, 0.56806474673115580251, 0.12053668025532305335,
      -0.35460488704253562597, -0.74851074817110109863, -0.97094181742605202716};
  static constexpr double s[] = {
      0.46472317204376854566, 0.82298386589365639458, 0.99270887409805399280,
      0.93501624268541482344, 0.66312265824079520238, 0.23931566428755776715};
};
// The same at any m: cos is even, sin odd about m = R / 2.
template <int R> __host__ __device__ constexpr double rot_c(int m) {
  return m % R == 0 ? 1.0 : (m % R <= (R - 1) / 2 ? Rot<R>::c[m % R - 1] : Rot<R>::c[R - m % R - 1]);
}
template <int R> __host__ __device__ constexpr double rot_s(int m) {
  return m % R == 0 ? 0.0 : (m % R <= (R - 1) / 2 ? Rot<R>::s[m % R - 1] : -Rot<R>::s[R - m % R - 1]);
}

__device__ __forceinline__ double2 swapc(double2 a) { return mk(a.y, a.x); }
__device__ __forceinline__ float2 swapc(float2 a) { return mk(a.y, a.x); }

// acc + a * c for a real constant c (split for complex64 data).
__device__ __forceinline__ double2 fma_r(double2 a, double c, double2 acc) {
  return mk(fma(a.x, c, acc.x), fma(a.y, c, acc.y));
}
__device__ __forceinline__ float2 fma_r(float2 a, double c, float2 acc) {
  const SplitF s = split_f(c);
  return mk(__fmaf_rn(a.x, s.hi, __fmaf_rn(a.x, s.lo, acc.x)),
            __fmaf_rn(a.y, s.hi, __fmaf_rn(a.y, s.lo, acc.y)));
}

// f(integral_constant<B>) .. f(integral_constant<E - 1>): loops whose index is
// a constant expression, so that every factor is an immediate.
template <int B, int E, typename F> __device__ __forceinline__ void static_for(F f) {
  if constexpr (B < E) {
    f(std::integral_constant<int, B>{});
    static_for<B + 1, E>(f);
  }
}

// Forward DFT of odd length R, unrolled: v is overwritten,
// output r goes to st(r, value).
template <int R, typename C, typename St>
__device__ __forceinline__ void dft_odd(C (&v)[R], St st) {
  constexpr int H = (R - 1) / 2;
  C sum = v[0];
#pragma unroll
  for (int j = 1; j <= H; ++j) {
    const C a = v[j], b = v[R - j];
    v[j] = cadd(a, b);
    v[R - j] = csub(a, b);
    sum = cadd(sum, v[j]);
  }
  st(0, sum);
  static_for<1, H + 1>([&](auto kc) {
    constexpr int k = decltype(kc)::value;
    C a = v[0], b{};
    static_for<1, H + 1>([&](auto jc) {
      constexpr int j = decltype(jc)::value;
      constexpr double c = rot_c<R>(j * k), s = rot_s<R>(j * k);
      a = fma_r(v[j], c, a);
      b = fma_r(v[R - j], s, b);
    });
    st(k, mk(a.x + b.y, a.y - b.x));
    st(R - k, mk(a.x - b.y, a.y + b.x));
  });
}

// Shared-memory accesses by 32-bit address: the passes below are functions of
// their own, in which a pointer would be a generic one.
__device__ __forceinline__ double2 lds(unsigned a, double2) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 lds(unsigned a, float2) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ float4 lds(unsigned a, float4) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a));
  return v;
}
__device__ __forceinline__ void sts(unsigned a, double2 v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void sts(unsigned a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}

// acc + a * (first or second part of a table entry).
__device__ __forceinline__ double2 fma_c(double2 a, double2 w, double2 acc) {
  return mk(fma(a.x, w.x, acc.x), fma(a.y, w.x, acc.y));
}
__device__ __forceinline__ double2 fma_s(double2 a, double2 w, double2 acc) {
  return mk(fma(a.x, w.y, acc.x), fma(a.y, w.y, acc.y));
}
__device__ __forceinline__ float2 fma_c(float2 a, float4 w, float2 acc) {
  return mk(__fmaf_rn(a.x, w.x, __fmaf_rn(a.x, w.z, acc.x)),
            __fmaf_rn(a.y, w.x, __fmaf_rn(a.y, w.z, acc.y)));
}
__device__ __forceinline__ float2 fma_s(float2 a, float4 w, float2 acc) {
  return mk(__fmaf_rn(a.x, w.y, __fmaf_rn(a.x, w.w, acc.x)),
            __fmaf_rn(a.y, w.y, __fmaf_rn(a.y, w.w, acc.y)));
}

// The same for the primes from 11 on, only the output pairs k0 .. k1 - 1 (and
// output 0 when k0 is 1): a loop over them with the factors from a table in
// shared memory, (cos, sin)(2 pi j k / R) at entry (k - 1) * H + j - 1.
// Unrolled over k as well, the code of one butterfly is so long that a line
// pass, which runs it once or twice a line, waits for instructions.
template <int R, typename C, typename St>
__device__ __forceinline__ void dft_prime(C (&v)[R], unsigned rot, int k0, int k1, St st) {
  constexpr int H = (R - 1) / 2;
  C sum = v[0];
#pragma unroll
  for (int j = 1; j <= H; ++j) {
    const C a = v[j], b = v[R - j];
    v[j] = cadd(a, b);
    v[R - j] = csub(a, b);
    sum = cadd(sum, v[j]);
  }
  if (k0 == 1) st(0, sum);
  rot += (unsigned)(k0 - 1) * (H * 16u);
#pragma unroll 1
  for (int k = k0; k < k1; ++k, rot += H * 16u) {
    C a = v[0], b{};
#pragma unroll
    for (int j = 1; j <= H; ++j) {
      const Tw<C> w = lds(rot + (unsigned)(j - 1) * 16u, Tw<C>{});
      a = fma_c(v[j], w, a);
      b = fma_s(v[R - j], w, b);
    }
    st(k, mk(a.x + b.y, a.y - b.x));
    st(R - k, mk(a.x - b.y, a.y + b.x));
  }
}

// v * exp(-2 pi i m / 9), split constants for complex64 data.
template <int M> __device__ __forceinline__ double2 w9(double2 v) {
  constexpr double c = rot_c<9>(M), s = -rot_s<9>(M);
  return mk(fma(v.x, c, -v.y * s), fma(v.x, s, v.y * c));
}
template <int M> __device__ __forceinline__ float2 w9(float2 v) {
  constexpr SplitF c = split_f(rot_c<9>(M)), s = split_f(-rot_s<9>(M));
  return tw_mul(v, make_float4(c.hi, s.hi, c.lo, s.lo));
}

// Forward DFT of length 9 as 3 x 3.
template <typename C, typename St> __device__ __forceinline__ void dft9(C (&v)[9], St st) {
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    C t[3] = {v[u], v[u + 3], v[u + 6]};
    dft_odd<3>(t, [&](int r, C x) { v[u + 3 * r] = x; });
  }
  v[4] = w9<1>(v[4]);
  v[5] = w9<2>(v[5]);
  v[7] = w9<2>(v[7]);
  v[8] = w9<4>(v[8]);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    C t[3] = {v[3 * q], v[3 * q + 1], v[3 * q + 2]};
    dft_odd<3>(t, [&](int r, C x) { st(q + 3 * r, x); });
  }
}

// One pass of radix R from x to y (shared addresses) by the TL threads lane =
// 0 .. TL - 1; tw, rot: the pass's twiddles and factors, in shared memory.  A
// butterfly of a large prime is shared by as many threads as there are to
// spare, each taking some of its output pairs (all read and fold the inputs).
// Not inlined: one copy a data type instead of one a kernel.
template <int R, typename C, bool UNROLL>
__device__ __noinline__ void pass(unsigned x, unsigned y, unsigned tw, unsigned rot, int nb, int ns,
                                  unsigned magic, int lane, int TL) {
  constexpr unsigned B = sizeof(C);
  constexpr int H = (R - 1) / 2;
  int split = 1, items = nb;
  if constexpr (R > 9 && R % 2 == 1 && !UNROLL) {
    split = TL / nb;
    split = split < 1 ? 1 : split > H ? H : split;
    items = nb * split;
  }
#pragma unroll 1
  for (int i = lane; i < items; i += TL) {
    int b = i, part = 0;
    if constexpr (R > 9 && R % 2 == 1 && !UNROLL) {
      while (b >= nb) {
        b -= nb;
        ++part;
      }
    }
    C v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = lds(x + (unsigned)(b + r * nb) * B, C{});
    int k = 0;
    if (ns > 1) {
      k = b - ns * (int)__umulhi((unsigned)b, magic);
#pragma unroll
      for (int r = 1; r < R; ++r)
        v[r] = tw_mul(v[r], lds(tw + (unsigned)((r - 1) * ns + k) * 16u, Tw<C>{}));
    }
    const unsigned o = y + (unsigned)((b - k) * R + k) * B;
    auto st = [&](int r, C val) { sts(o + (unsigned)(r * ns) * B, val); };
    if constexpr (R == 9) {
      dft9(v, st);
    } else if constexpr (R > 9 && R % 2 == 1 && !UNROLL) {
      dft_prime<R>(v, rot, 1 + part * H / split, 1 + (part + 1) * H / split, st);
    } else if constexpr (R % 2 == 1) {
      dft_odd<R>(v, st);
    } else {
      dft_r<R, -1>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) st(r, v[r]);
    }
  }
}

// Forward transform of the line in a (length plan.n) by TL threads; b: the
// second buffer, tws: the plan's table in shared memory.  Returns the buffer
// that holds the result.  sync() orders the TL threads; the caller has
// synchronised after writing a, the transform synchronises after its last
// pass.  BIG: radices above 13 may occur (they set the register count).  HOT:
// the same line is transformed over and over, so the code stays in the
// instruction cache and 11 and 13 are unrolled.
template <bool BIG, bool HOT, typename C, typename Sync>
__device__ __forceinline__ C *transform(C *a, C *b, const Tw<C> *tws, const MixedPlan &plan,
                                        int lane, int TL, Sync sync) {
  int ns = 1;
  const unsigned tab = (unsigned)__cvta_generic_to_shared(tws);
  unsigned tw = tab;
  unsigned x = (unsigned)__cvta_generic_to_shared(a), y = (unsigned)__cvta_generic_to_shared(b);
  MixedPlan::Pass ps = plan.pass[0];
#pragma unroll 1
  for (int p = 0; p < plan.passes; ++p) {
    const int r = ps.radix, nb = ps.nb;
    const unsigned magic = ps.magic, rot = tab + 16u * (unsigned)ps.rot;
#define PXP_MIXED_PASS(RR)                                                          \
  case RR:                                                                          \
    pass<RR, C, (HOT && RR <= 13)>(x, y, tw, rot, nb, ns, magic, lane, TL);          \
    break;
    switch (r) {
      PXP_MIXED_PASS(2) PXP_MIXED_PASS(3) PXP_MIXED_PASS(4) PXP_MIXED_PASS(5) PXP_MIXED_PASS(7)
      PXP_MIXED_PASS(8) PXP_MIXED_PASS(9) PXP_MIXED_PASS(11) PXP_MIXED_PASS(13)
      default:
        if constexpr (BIG) {
          switch (r) {
            PXP_MIXED_PASS(17) PXP_MIXED_PASS(19) PXP_MIXED_PASS(23) PXP_MIXED_PASS(29)
            PXP_MIXED_PASS(31)
            default: break;
          }
        }
    }
#undef PXP_MIXED_PASS
    if (p + 1 < plan.passes) ps = plan.pass[p + 1];
    sync();
    tw += (unsigned)((r - 1) * ns) * 16u;
    ns *= r;
    const unsigned t = x;
    x = y;
    y = t;
  }
  return plan.passes & 1 ? b : a;
}

}  // namespace mixed
}  // namespace pxp
