// mixed_plan.h -- the plan of a mixed-radix transform (host and device, no CUDA
// headers).
#pragma once

namespace pxp {

// Passes of the mixed-radix transform (fft_mixed.cuh) of length n, in order:
// radix, butterflies (n / radix), the multiplier that divides a butterfly's
// index by the pass's sub-transform length, and for radices above 9 where
// their (cos, sin) factors lie in the table (16 bytes: one load a pass).
struct MixedPlan {
  static constexpr int kMaxPasses = 8;
  struct alignas(16) Pass {
    int radix, nb;
    unsigned magic;
    int rot;
  };
  Pass pass[kMaxPasses];
  int n, passes;
  int table;  // entries of the table
  bool big;   // a radix above 13
};
// Fills *plan (may be null) and returns true for lengths that are not powers
// of two and have no prime factor above 31.
bool mixed_plan(int n, MixedPlan *plan);

// Line passes (fft3d_mixed.cu): threads a line and lines a CTA.  Short lines one a
// CTA (300 nodes: 14.8 us a step against 17.8 with two of 64 threads); around
// 513 nodes, whose primes give a pass few butterflies, 64 threads (29 us; 128:
// 39); above, complex64 lines keep 64 threads (1000: 49 us; 128: 57), complex128
// lines take 128 (61 us; 64: 73), two a CTA while both fit shared memory.
struct MixedLines {
  int threads, lines;
};
inline MixedLines mixed_lines(int n, bool complex64) {
  if (n <= 400) return {128, 1};
  if (n <= (complex64 ? 1200 : 700)) return {64, 2};
  return n <= 2700 ? MixedLines{128, 2} : MixedLines{256, 1};
}
// Their shared memory: two buffers a line and the table.
inline unsigned long long mixed_lines_smem(const MixedPlan &plan, int lines, bool complex64) {
  return 2ull * (complex64 ? 8 : 16) * lines * plan.n + 16ull * plan.table;
}

}  // namespace pxp
