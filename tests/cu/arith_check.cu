// The reciprocal and the division by a constant of pxp_complex.cuh against the
// correctly rounded 1.0 / m and a / s, on the device.  Prints the largest
// differences in units of the last place and the number of mismatches.
#include <cstdio>
#include <cstring>

#include "../../paxpro_b200/csrc/pxp_complex.cuh"

using namespace pxp;

__device__ unsigned long long mix(unsigned long long x) {  // splitmix64
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}
// A double with the given biased exponent and random significand and sign bits.
__device__ double draw(unsigned long long seed, int exponent, bool sign) {
  const unsigned long long b = mix(seed);
  return __longlong_as_double((long long)((b >> 12) | ((unsigned long long)exponent << 52) |
                                          (sign ? b << 63 : 0ull)));
}
__device__ unsigned long long ulps(double a, double b) {
  const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
  return x > y ? (unsigned long long)(x - y) : (unsigned long long)(y - x);
}

// [0] largest difference of rcp_newton over its range; [1] values wrong at its ends;
// [2] div_by: normal results that differ; [3] largest difference of subnormal
// ones; [4] special values wrong, or the two forms of the division differ
__global__ void check(unsigned long long *out) {
  const unsigned long long id = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
  // every exponent whose reciprocal is normal: 2^-1022 <= m <= 2^1022
  for (int e = 1; e < 2045; ++e) {
    const double m = draw(id * 4096 + e, e, false);
    atomicMax(out, ulps(rcp_newton(m), __drcp_rn(m)));
  }
  const double inf = __longlong_as_double(0x7ff0000000000000ll);
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const double huge = 1.7976931348623157e308, tiny = 2.2250738585072014e-308, sub = 4.9e-324;
  if (id == 0) {
    bool bad = rcp_newton(nan) == rcp_newton(nan) || rcp_newton(1.0 / tiny) != tiny ||
               rcp_newton(1.0) != 1.0 || rcp_newton(tiny) != __drcp_rn(tiny);
    if (bad) atomicAdd(out + 1, 1ull);
  }
  // lengths n and n * n
  for (int k = 0; k < 64; ++k) {
    const double n = (double)(3 + (id * 64 + k) % 8190), s = k & 1 ? n * n : n;
    const Divisor d = divisor(s);
    for (int e = 1; e < 2047; e += 7) {
      const double a = draw((id * 64 + k) * 4096 + e, e, true);
      const double got = div_by(a, d), want = __ddiv_rn(a, s);
      if (ulps(got, div_by_tested(a, d))) atomicAdd(out + 4, 1ull);
      if (fabs(want) >= tiny) {
        if (ulps(got, want)) atomicAdd(out + 2, 1ull);
      } else {
        atomicMax(out + 3, ulps(got, want));
      }
    }
    const double z = draw(id * 64 + k, 0, true);  // a subnormal
    atomicMax(out + 3, ulps(div_by(z, d), __ddiv_rn(z, s)));
    const double special[] = {0.0, -0.0, inf, -inf, huge, -huge, sub, -sub, tiny, -tiny};
    for (double a : special)
      if (ulps(div_by(a, d), __ddiv_rn(a, s)) || ulps(div_by_tested(a, d), __ddiv_rn(a, s)))
        atomicAdd(out + 4, 1ull);
    if (div_by(nan, d) == div_by(nan, d) || div_by_tested(nan, d) == div_by_tested(nan, d))
      atomicAdd(out + 4, 1ull);
  }
}

int main() {
  unsigned long long *d, h[5] = {};
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMemset(d, 0, sizeof(h)) != cudaSuccess) return 2;
  check<<<296, 128>>>(d);
  if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("rcp %llu %llu div %llu %llu %llu\n", h[0], h[1], h[2], h[3], h[4]);
  return 0;
}
