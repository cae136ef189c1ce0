// fft1d_r8.cu -- FFTSolver2D split step with register-resident radix-8
// transforms (powers of two from 64 to 2048 points, complex64 to 4096), 8
// points and n/8 threads a line.
//
// The step of fft1d_r16.cu with half the points a thread: thread j holds the
// points j + s*n/8 (s = 0 .. 7) for the whole launch; a transform is a first
// pass of radix R0 = 8, 4 or 2 on the thread's own points (n = R0 * 8^k) and k
// radix-8 Stockham passes through two alternating exchange buffers, one
// barrier a pass (a warp barrier up to 256 points).  A thread's twiddles are
// the same in every step, so they stay in registers, as does the propagator.
// A single line is bound by latency on one SM; spreading it over twice the
// warps shortens each thread's chain at the price of one more exchange than
// radix 16 from 1024 points on.  Measured, us a step (a single problem; before:
// the faster of the shared-memory kernel and radix 16): FP64 256 points 2.2 ->
// 1.1, 512: 1.99 -> 1.03, 1024: 2.12 -> 1.61, 2048: 3.39 -> 2.65; FP32 512: 1.72
// -> 0.75, 1024: 3.6 -> 1.09, 2048: 4.0 -> 1.87, 4096: 4.5 -> 4.0.  With more
// problems than SMs (444 of one size, us a step, problem and SM): FP32 512
// 1.16 -> 0.82, 2048: 2.44 -> 2.24; FP64 2048 2.99 -> 2.95.
#include "fft_smem.cuh"
#include "flux.cuh"
#include "persistent.cuh"
#include "pxp_kernels.h"

namespace pxp {
namespace r8_1d {

constexpr int log2c(int n) { return n <= 1 ? 0 : 1 + log2c(n / 2); }
template <int N> struct Plan {
  static constexpr int LOG = log2c(N);
  static constexpr int R0 = 1 << (LOG % 3 == 0 ? 3 : LOG % 3);
  static constexpr int NP = (LOG - log2c(R0)) / 3;  // radix-8 passes
  static constexpr int TL = N / 8;
  // Twiddles: in registers for every pass up to 2048 points (the propagator
  // too); at 4096 a thread has 128 registers, and only the last pass's stay
  // there, the earlier passes' few distinct values (R0 * (8^(NP-1) - 1)) being
  // read from shared memory.
  static constexpr bool ALL_REG = N <= 2048;
  static constexpr int NPR = ALL_REG ? NP : 1;
  static constexpr int TWS = ALL_REG ? 0 : R0 * ((1 << (3 * (NP - 1))) - 1);
};

// A thread's twiddles.
template <int N, typename W> struct Twiddles {
  W reg[Plan<N>::NPR][7];
  const W *smem;
  template <int P> __device__ __forceinline__ W at(int r, int j) const {
    constexpr int FIRST = Plan<N>::NP - Plan<N>::NPR;
    if constexpr (P >= FIRST) {
      return reg[P - FIRST][r - 1];
    } else {
      constexpr int NS = Plan<N>::R0 << (3 * P);
      constexpr int OFF = Plan<N>::R0 * ((1 << (3 * P)) - 1);  // 7 NS entries a pass
      return smem[OFF + (r - 1) * NS + (j & (NS - 1))];
    }
  }
};

__device__ __forceinline__ double2 refract(double2 u, double2 t, double inv_n) {
  return cx_scale_rn(cx_mul_rn(u, t), inv_n);  // N a power of two: as the division rounds
}
__device__ __forceinline__ float2 refract(float2 u, float4 t, float) { return tw_mul(u, t); }
__device__ __forceinline__ double2 kmul(double2 u, double2 k) { return cx_mul_rn(u, k); }
__device__ __forceinline__ float2 kmul(float2 u, float4 k) { return tw_mul(u, k); }

template <int TL> __device__ __forceinline__ void line_sync() {
  if constexpr (TL <= 32) __syncwarp(TL >= 32 ? 0xffffffffu : (1u << TL) - 1u);
  else __syncthreads();
}

// Radix-8 pass P of a transform: read at stride TL, twiddles, DFT; unless it
// is the last pass, write to the other buffer for the next one.
template <int SIGN, int N, int P, typename C>
__device__ __forceinline__ void passes(C (&v)[8], C *x, C *y, const Twiddles<N, Tw<C>> &tw, int j) {
  constexpr int TL = Plan<N>::TL;
  line_sync<TL>();
#pragma unroll
  for (int r = 0; r < 8; ++r) v[r] = x[sw<C>(j + r * TL)];
#pragma unroll
  for (int r = 1; r < 8; ++r) {
    const Tw<C> w = tw.template at<P>(r, j);
    v[r] = SIGN < 0 ? tw_mul(v[r], w) : tw_mulc(v[r], w);
  }
  dft8<SIGN>(v);
  if constexpr (P + 1 < Plan<N>::NP) {
    constexpr int NS = Plan<N>::R0 << (3 * P);
    const int k = j & (NS - 1), base = (j - k) * 8 + k;
#pragma unroll
    for (int r = 0; r < 8; ++r) y[sw<C>(base + r * NS)] = v[r];
    passes<SIGN, N, P + 1>(v, y, x, tw, j);
  }
}

// One transform of the thread's 8 points, natural order before and after.
// X0, X1: with NP passes the first is written to x and read from it; a
// buffer is written again only after a barrier that follows its last read
// (the next transform starts with the buffer this one did not end on).
template <int SIGN, int N, typename C>
__device__ __forceinline__ void line_fft(C (&v)[8], C *x, C *y, const Twiddles<N, Tw<C>> &tw, int j) {
  constexpr int R0 = Plan<N>::R0, TL = Plan<N>::TL;
#pragma unroll
  for (int u = 0; u < 8 / R0; ++u) {
    C w[R0];
#pragma unroll
    for (int r = 0; r < R0; ++r) w[r] = v[u + r * (8 / R0)];
    dft_r<R0, SIGN>(w);
#pragma unroll
    for (int r = 0; r < R0; ++r) x[sw<C>((j + u * TL) * R0 + r)] = w[r];
  }
  passes<SIGN, N, 0>(v, x, y, tw, j);
}

template <typename R, int N, bool FLUX>
__global__ void __launch_bounds__(N / 8) fft1d_r8_kernel(const Fft1dJob *__restrict__ jobs,
                                                        int step0_ov, int nsteps_ov, int njobs,
                                                        unsigned *queue) {
  using C = typename Cx<R>::T;
  using W = Tw<C>;
  using P = Plan<N>;
  constexpr int TL = P::TL;
  // the transforms of a step start on alternating buffers: with an odd number
  // of passes a transform ends on the buffer it started with
  constexpr bool ODD = P::NP % 2 == 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double flux_red[2][flux_slots<TL>()];
  __shared__ int s_next;
  C *X0 = reinterpret_cast<C *>(smem_raw);
  C *X1 = X0 + N;
  for (int jb = blockIdx.x; jb < njobs; jb = next_job(queue, &s_next)) {
    Fft1dJob job = jobs[jb];
    if (nsteps_ov >= 0) {
      job.step0 = step0_ov;
      job.nsteps = nsteps_ov;
    }
    const int j = threadIdx.x;
    Twiddles<N, W> tw;
    const W *wn = reinterpret_cast<const W *>(job.wn);
    constexpr int FIRST = P::NP - P::NPR;
    if constexpr (!P::ALL_REG) {
      W *tws = reinterpret_cast<W *>(X1 + N);
      tw.smem = tws;
      for (int p = 0, ns = P::R0, off = 0; p < FIRST; ++p, off += 7 * ns, ns *= 8)
        for (int i = j; i < 7 * ns; i += TL)
          tws[off + i] = wn[(i / ns + 1) * (i % ns) * (N / (8 * ns))];
      __syncthreads();
    }
#pragma unroll
    for (int p = FIRST, ns = P::R0 << (3 * FIRST); p < P::NP; ++p, ns *= 8)
#pragma unroll
      for (int r = 1; r < 8; ++r) tw.reg[p - FIRST][r - 1] = wn[r * (j & (ns - 1)) * (N / (8 * ns))];
    const W *kern = reinterpret_cast<const W *>(job.kern);
    W kp[8];
    if constexpr (P::ALL_REG)
#pragma unroll
      for (int s = 0; s < 8; ++s) kp[s] = kern[j + s * TL];
    C *field = reinterpret_cast<C *>(job.field);
    C v[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) v[s] = field[j + s * TL];
    const W *trans0 = reinterpret_cast<const W *>(job.trans);
    C *saves = reinterpret_cast<C *>(job.saves);
    for (int st = 0; st < job.nsteps; ++st) {
      const int step = job.step0 + st;
      int2 fw;
      const bool flux = FLUX && flux_window(job.flux, step, fw);
      line_fft<-1, N>(v, X0, X1, tw, j);
#pragma unroll
      for (int s = 0; s < 8; ++s)
        v[s] = kmul(v[s], P::ALL_REG ? kp[s] : __ldg(kern + j + s * TL));
      const W *trans = trans0 + job.trans_stride * (long long)(step - job.trans_step0);
      W t[8];
      if constexpr (P::ALL_REG)
#pragma unroll
        for (int s = 0; s < 8; ++s) t[s] = __ldg(trans + j + s * TL);
      if constexpr (ODD) line_fft<+1, N>(v, X1, X0, tw, j);
      else line_fft<+1, N>(v, X0, X1, tw, j);
      const bool save = job.save_every > 0 && saves != nullptr && (step % job.save_every) == 0 &&
                        (step / job.save_every - 1) < job.max_slots;
      C *slot = save ? saves + (long long)(step / job.save_every - 1) * N : nullptr;
      double acc = 0.0;
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const int e = j + s * TL;
        v[s] = refract(v[s], P::ALL_REG ? t[s] : __ldg(trans + e), (R)1 / (R)N);
        if (save) slot[e] = v[s];
        if (flux) flux_add(acc, e, fw, to_d(v[s]));
      }
      if constexpr (FLUX) {
        if (flux) flux_warp_total<TL>(acc, flux_red[st & 1]);
        __syncthreads();
        if (flux) flux_store<TL>(job.flux, step, flux_red[st & 1]);
      }
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) field[j + s * TL] = v[s];
  }
}

template <typename R, int N, bool FLUX>
cudaError_t launch(const Fft1dJob *d_jobs, int nj, int step0, int nsteps, cudaStream_t s,
                   unsigned *queue) {
  using C = typename Cx<R>::T;
  constexpr size_t smem = 2 * sizeof(C) * N + sizeof(Tw<C>) * Plan<N>::TWS;
  auto k = fft1d_r8_kernel<R, N, FLUX>;
  const cudaError_t e = raise_dynamic_smem((const void *)k, (int)smem);
  if (e != cudaSuccess) return e;
  const int grid = persistent_grid((const void *)k, N / 8, smem, nj, queue);
  k<<<grid, N / 8, smem, s>>>(d_jobs, step0, nsteps, nj, queue);
  return cudaGetLastError();
}

}  // namespace r8_1d

bool fft1d_r8_enabled(Precision p, int n) {
  return n >= 64 && n <= (p == kFP64 ? 2048 : 4096) && !(n & (n - 1));
}

cudaError_t launch_fft1d_r8(Precision p, const Fft1dJob *d_jobs, int nj, int n, int step0,
                            int nsteps, cudaStream_t s, bool flux, unsigned *queue) {
#define PXP_1R(NN)                                                                          \
  case NN:                                                                                  \
    if (p == kFP64)                                                                         \
      return flux ? r8_1d::launch<double, NN, true>(d_jobs, nj, step0, nsteps, s, queue)    \
                  : r8_1d::launch<double, NN, false>(d_jobs, nj, step0, nsteps, s, queue);  \
    return flux ? r8_1d::launch<float, NN, true>(d_jobs, nj, step0, nsteps, s, queue)       \
                : r8_1d::launch<float, NN, false>(d_jobs, nj, step0, nsteps, s, queue);
  switch (n) {
    PXP_1R(64) PXP_1R(128) PXP_1R(256) PXP_1R(512) PXP_1R(1024) PXP_1R(2048)
    case 4096:
      if (p != kFP32) return cudaErrorInvalidValue;
      return flux ? r8_1d::launch<float, 4096, true>(d_jobs, nj, step0, nsteps, s, queue)
                  : r8_1d::launch<float, 4096, false>(d_jobs, nj, step0, nsteps, s, queue);
    default:
      return cudaErrorInvalidValue;
  }
#undef PXP_1R
}

}  // namespace pxp
