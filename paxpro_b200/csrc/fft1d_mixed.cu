// fft1d_mixed.cu -- FFTSolver2D split step for lengths that are not powers of
// two and whose prime factors are at most 31 (the reference plans FFTW for any
// length, src/fftSolver2D.cpp:68-69); other lengths use the chirp-z kernel of
// fft1d.cu.
//
// One CTA per problem keeps the field in shared memory for all steps of the
// launch.  A step is two mixed-radix transforms (fft_mixed.cuh) and two
// pointwise loops: propagator, then refraction, saves and flux terms, with
// the arithmetic of fft1d.cu.  What bounds it: the latency of one SM's serial
// passes -- a barrier each, few butterflies of long chains (77 of 13 points at
// 1001) -- not its FP64 rate (18 % of the pipe).  Table and field stay in
// shared memory.  Measured against the chirp-z kernel (us a step, FP64): 300
// points 10.3 -> 3.2, 600: 10.5 -> 3.9, 1001: 11.4 -> 4.7, 3000: 55 -> 11.7; FP32
// 1000: 8.4 -> 4.2.
#include "fft_mixed.cuh"
#include "flux.cuh"

namespace pxp {

bool mixed_plan(int n, MixedPlan *plan) {
  static const int kOdd[] = {31, 29, 23, 19, 17, 13, 11, 9, 7, 5, 3};
  MixedPlan p{};
  p.n = n;
  // two buffers and the table fit shared memory up to 4096 points
  if (n < 2 || n > 4096 || !(n & (n - 1))) return false;
  int rest = n, ns = 1;
  p.table = n - 1;
  auto add = [&](int r) {
    MixedPlan::Pass &q = p.pass[p.passes];
    q.radix = r;
    q.nb = n / r;
    // floor(b / ns) = b * magic >> 32 for b < 2^16
    q.magic = ns > 1 ? (unsigned)((0x100000000ull + ns - 1) / ns) : 0u;
    if (r > 9) {
      const bool again = p.passes > 0 && p.pass[p.passes - 1].radix == r;
      q.rot = again ? p.pass[p.passes - 1].rot : p.table;
      if (!again) p.table += (r / 2) * (r / 2);
    }
    ++p.passes;
    ns *= r;
    rest /= r;
  };
  for (int r : kOdd)
    while (rest % r == 0) {
      if (p.passes == MixedPlan::kMaxPasses) return false;
      p.big = p.big || r > 13;
      add(r);
    }
  for (int r : {8, 4, 2})
    while (rest % r == 0 && rest > 1) {
      if (p.passes == MixedPlan::kMaxPasses) return false;
      add(r);
    }
  if (rest != 1) return false;
  if (plan) *plan = p;
  return true;
}

namespace {

__device__ __forceinline__ void refract(double2 &u, double2 t, Divisor n) {
  u = cx_div_by(cx_mul_rn(u, t), n);
}
__device__ __forceinline__ void refract(float2 &u, float4 t, Divisor) { u = tw_mul(u, t); }
__device__ __forceinline__ double2 kmul(double2 u, double2 k) { return cx_mul_rn(u, k); }
__device__ __forceinline__ float2 kmul(float2 u, float4 k) { return tw_mul(u, k); }

constexpr int kMaxT = 256;

// f(i, ld(i), tab(i)) for i = lane, lane + T, ... below n, the loads of four
// points in flight at a time (in a plain loop each point's store holds back
// the next point's load from the same buffer).
template <typename Ld, typename Tab, typename F>
__device__ __forceinline__ void for_points(int lane, int n, int T, Ld ld, Tab tab, F f) {
  for (int i0 = lane; i0 < n; i0 += 4 * T) {
    decltype(ld(0)) v[4];
    decltype(tab(0)) w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * T < n) {
        v[u] = ld(i0 + u * T);
        w[u] = tab(i0 + u * T);
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * T < n) f(i0 + u * T, v[u], w[u]);
  }
}

template <typename R, bool BIG, bool FLUX>
__global__ void __launch_bounds__(kMaxT)
    fft1d_mixed_kernel(const Fft1dJob *__restrict__ jobs, const __grid_constant__ MixedPlan plan,
                       int step0_ov, int nsteps_ov) {
  using C = typename Cx<R>::T;
  using W = Tw<C>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double flux_red[2][flux_slots<kMaxT>()];
  const int n = plan.n, lane = threadIdx.x, T = blockDim.x;
  if (lane < 2 * flux_slots<kMaxT>()) (&flux_red[0][0])[lane] = 0.0;  // the slots of warps not launched
  Fft1dJob job = jobs[blockIdx.x];
  if (nsteps_ov >= 0) {
    job.step0 = step0_ov;
    job.nsteps = nsteps_ov;
  }
  const W *tw = reinterpret_cast<const W *>(job.twiddle);
  W *stw = reinterpret_cast<W *>(smem_raw);
  for (int i = lane; i < plan.table; i += T) stw[i] = tw[i];
  tw = stw;
  C *a = reinterpret_cast<C *>(stw + plan.table);
  C *b = a + n;
  C *field = reinterpret_cast<C *>(job.field);
  for (int i = lane; i < n; i += T) a[i] = field[i];
  __syncthreads();
  const W *kern = reinterpret_cast<const W *>(job.kern);
  const W *trans0 = reinterpret_cast<const W *>(job.trans);
  C *saves = reinterpret_cast<C *>(job.saves);
  const Divisor nreal = divisor((double)n);
  auto sync = [] { __syncthreads(); };
  for (int s = 0; s < job.nsteps; ++s) {
    const int step = job.step0 + s;
    int2 fw;
    const bool flux = FLUX && flux_window(job.flux, step, fw);
    C *x = mixed::transform<BIG, true>(a, b, tw, plan, lane, T, sync);
    C *y = x == a ? b : a;
    for_points(lane, n, T, [&](int i) { return x[i]; }, [&](int i) { return __ldg(kern + i); },
               [&](int i, C v, W w) { x[i] = mixed::swapc(kmul(v, w)); });
    __syncthreads();
    a = mixed::transform<BIG, true>(x, y, tw, plan, lane, T, sync);
    b = a == x ? y : x;
    const W *trans = trans0 + job.trans_stride * (long long)(step - job.trans_step0);
    const bool save = job.save_every > 0 && saves != nullptr && (step % job.save_every) == 0 &&
                      (step / job.save_every - 1) < job.max_slots;
    C *slot = save ? saves + (long long)(step / job.save_every - 1) * n : nullptr;
    double acc = 0.0;
    for_points(lane, n, T, [&](int i) { return mixed::swapc(a[i]); },
               [&](int i) { return __ldg(trans + i); },
               [&](int i, C v, W w) {
                 refract(v, w, nreal);
                 a[i] = v;
                 if (save) slot[i] = v;
                 if (flux) flux_add(acc, i, fw, to_d(v));
               });
    if (flux) flux_warp_total<kMaxT>(acc, flux_red[s & 1]);
    __syncthreads();
    if (flux) flux_store<kMaxT>(job.flux, step, flux_red[s & 1]);
  }
  for (int i = lane; i < n; i += T) field[i] = a[i];
}

template <typename R, bool BIG, bool FLUX>
cudaError_t launch_t(const Fft1dJob *d_jobs, const MixedPlan &plan, int nj, int step0, int nsteps,
                     cudaStream_t s) {
  const size_t smem = 2 * sizeof(typename Cx<R>::T) * plan.n + 16 * (size_t)plan.table;
  if (smem > 225 * 1024) return cudaErrorInvalidValue;  // mixed_plan bounds n
  auto k = fft1d_mixed_kernel<R, BIG, FLUX>;
  const cudaError_t e = raise_dynamic_smem((const void *)k, (int)smem);
  if (e != cudaSuccess) return e;
  // 300 points: 160 threads 3.15 us a step, 256 3.25; 1001: 9.4 / 4.9 / 4.7 us
  // at 64 / 160 / 256; 3000: 14.4 / 13.8 / 11.7 us at 128 / 160 / 256
  const int T = plan.n <= 400 ? 160 : kMaxT;
  k<<<nj, T, smem, s>>>(d_jobs, plan, step0, nsteps);
  return cudaGetLastError();
}

template <typename R>
cudaError_t launch_r(const Fft1dJob *d_jobs, const MixedPlan &plan, int nj, int step0, int nsteps,
                     cudaStream_t s, bool flux) {
  if (plan.big)
    return flux ? launch_t<R, true, true>(d_jobs, plan, nj, step0, nsteps, s)
                : launch_t<R, true, false>(d_jobs, plan, nj, step0, nsteps, s);
  return flux ? launch_t<R, false, true>(d_jobs, plan, nj, step0, nsteps, s)
              : launch_t<R, false, false>(d_jobs, plan, nj, step0, nsteps, s);
}

}  // namespace

cudaError_t launch_fft1d_mixed(Precision p, const Fft1dJob *d_jobs, int nj, int n, int step0,
                               int nsteps, cudaStream_t s, bool flux) {
  MixedPlan plan;
  if (!mixed_plan(n, &plan)) return cudaErrorInvalidValue;
  return p == kFP64 ? launch_r<double>(d_jobs, plan, nj, step0, nsteps, s, flux)
                    : launch_r<float>(d_jobs, plan, nj, step0, nsteps, s, flux);
}

}  // namespace pxp
