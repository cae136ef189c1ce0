// fft3d_mixed.cu -- FFTSolver3D line passes for grid sizes that are not powers
// of two and whose prime factors are at most 31 (the reference plans FFTW for
// any n, src/fftSolver3D.cpp:61-62; its own example grid has 513 = 19 * 27
// nodes, Examples/sphere.cpp:40); other sizes run fft3d_blu.cu.
//
// The same two passes per step as fft3d.cu (x pass: F_x, K, F_x^-1; y pass:
// F_y^-1, refraction, F_y), each line transform mixed-radix (fft_mixed.cuh).
// A CTA holds L adjacent lines, TL threads each, in two buffers a line; the
// line's threads synchronise among themselves only (a named
// barrier), so lines drift apart and one's loads cover another's arithmetic.
// Lines come and go cooperatively: contiguous lines as whole runs, strided
// ones as L adjacent elements a position.
// What bounds it: latency with 4 to 8 warps an SM (513 lines are 3.5 an SM);
// the field is L2-resident at these sizes.  Measured against the chirp-z
// kernel (us a step, FP64): 100 nodes 26 -> 12, 300: 38 -> 15, 513: 84 -> 29,
// 1000: 177 -> 61, 2001: 746 -> 364; FP32 551: 65 -> 30, 1000: 134 -> 51.
#include "fft3d_point.cuh"
#include "fft_mixed.cuh"

namespace pxp {
namespace {

template <int BYTES> __device__ __forceinline__ void copy_async(void *dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "n"(BYTES)
               : "memory");
}

template <typename R, int TL, int L, bool BIG>
__global__ void __launch_bounds__(TL *L) fft3d_mixed_kernel(const __grid_constant__ Fft3dPass q,
                                                           const __grid_constant__ MixedPlan plan,
                                                           const double *__restrict__ kx2) {
  using C = typename Cx<R>::T;
  using W = Tw<C>;
  constexpr int T = TL * L;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  W *tws = reinterpret_cast<W *>(smem_raw);            // the plan's table
  C *buf = reinterpret_cast<C *>(tws + plan.table);  // L x 2 x n
  const int n = plan.n;
  const int tid = threadIdx.x, slot = tid / TL, lane = tid % TL;
  const int line0 = blockIdx.x * L, line = line0 + slot;
  const int nl = n - line0 < L ? n - line0 : L;  // lines of this CTA
  C *field = reinterpret_cast<C *>(q.field);
  const bool strided = q.mode == 1;  // x lines: fixed row, stride n
  auto sync = [slot] { asm volatile("bar.sync %0, %1;\n" ::"r"(1 + slot), "n"(TL) : "memory"); };

  // the table does not depend on the previous kernel: copied while it drains
  for (int i = tid; i < plan.table; i += T)
    copy_async<16>(tws + i, reinterpret_cast<const W *>(q.twiddle) + i);
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (strided) {
    const int g = tid % L;
    if (g < nl)
      for (int p = tid / L; p < n; p += TL)
        copy_async<sizeof(C)>(buf + g * 2 * n + p, field + (long long)p * n + line0 + g);
  } else if (slot < nl) {
    for (int p = lane; p < n; p += TL)
      copy_async<sizeof(C)>(buf + slot * 2 * n + p, field + (long long)line * n + p);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();

  C *a = buf + slot * 2 * n, *b = a + n;
  if (slot < nl) {
    auto fft = [&] {
      C *x = mixed::transform<BIG, false>(a, b, tws, plan, lane, TL, sync);
      if (x != a) {
        b = a;
        a = x;
      }
    };
    if (q.mode == 1) {
      fft();
      const double ky = kfreq(line, n, q.two_pi, q.stepn_y);
      const double ky2 = __dmul_rn(ky, ky);
      for (int j0 = lane; j0 < n; j0 += 4 * TL) {
        C v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (const int j = j0 + u * TL; j < n) v[u] = mixed::swapc(prop3(q, a[j], kx2[j], ky2, j, line));
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (const int j = j0 + u * TL; j < n) a[j] = v[u];
      }
      sync();
      fft();
    } else {
      if (q.mode >= 2) {
        for (int j = lane; j < n; j += TL) a[j] = mixed::swapc(a[j]);
        sync();
        fft();
        C *save = reinterpret_cast<C *>(q.save);
        for (int j = lane; j < n; j += TL) {
          const C v = refract3<R>(q, mixed::swapc(a[j]), line, j, 0.0);  // 0: divide by n*n
          a[j] = v;
          if (save) save[(long long)line * n + j] = v;
        }
        sync();
      }
      if (q.mode != 3) fft();
    }
  }
  if (strided) {
    __syncthreads();
    const int g = tid % L;
    const C *r = buf + g * 2 * n;  // two transforms: back in the slot's first buffer
    if (g < nl)
      for (int p = tid / L; p < n; p += TL)
        field[(long long)p * n + line0 + g] = mixed::swapc(r[p]);
  } else if (slot < nl) {
    for (int p = lane; p < n; p += TL) field[(long long)line * n + p] = a[p];
  }
}

template <typename R, int TL, int L, bool BIG>
cudaError_t launch_t(const Fft3dPass &q, const MixedPlan &plan, const double *kx2, cudaStream_t s) {
  const size_t smem = mixed_lines_smem(plan, L, sizeof(R) == 4);
  if (smem > 227 * 1024) return cudaErrorInvalidValue;
  auto k = fft3d_mixed_kernel<R, TL, L, BIG>;
  const cudaError_t e = raise_dynamic_smem((const void *)k, (int)smem);
  if (e != cudaSuccess) return e;
  // a programmatic dependent of the previous kernel in the stream: its CTAs
  // start while that kernel drains and wait for it with griddepcontrol.wait
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((plan.n + L - 1) / L);
  cfg.blockDim = dim3(TL * L);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute la[1];
  la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  la[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = la;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, q, plan, kx2);
}

template <typename R, int TL, int L>
cudaError_t launch_b(const Fft3dPass &q, const MixedPlan &plan, const double *kx2, cudaStream_t s) {
  return plan.big ? launch_t<R, TL, L, true>(q, plan, kx2, s)
                  : launch_t<R, TL, L, false>(q, plan, kx2, s);
}

template <typename R>
cudaError_t launch_r(const Fft3dPass &q, const MixedPlan &plan, const double *kx2, cudaStream_t s) {
  const MixedLines l = mixed_lines(plan.n, sizeof(R) == 4);
  if (l.lines == 2)
    return l.threads == 64 ? launch_b<R, 64, 2>(q, plan, kx2, s) : launch_b<R, 128, 2>(q, plan, kx2, s);
  return l.threads == 128 ? launch_b<R, 128, 1>(q, plan, kx2, s) : launch_b<R, 256, 1>(q, plan, kx2, s);
}

}  // namespace

cudaError_t launch_fft3d_mixed(Precision p, const Fft3dPass &q, const double *kx2, cudaStream_t s) {
  MixedPlan plan;
  if (!mixed_plan(q.n, &plan)) return cudaErrorInvalidValue;
  return p == kFP64 ? launch_r<double>(q, plan, kx2, s) : launch_r<float>(q, plan, kx2, s);
}

}  // namespace pxp
