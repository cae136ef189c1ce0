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

}  // namespace pxp
