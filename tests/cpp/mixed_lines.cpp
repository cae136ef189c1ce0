// The line passes' launch shapes of every length the mixed-radix plan takes,
// checked without a GPU: whole warps, and shared memory that a CTA can have.
#include <cstdio>

#include "../../paxpro_b200/csrc/mixed_plan.h"

int main() {
  unsigned long long most = 0;
  for (int n = 2; n <= 4096; ++n) {
    pxp::MixedPlan p;
    if (!pxp::mixed_plan(n, &p)) continue;
    for (int complex64 = 0; complex64 < 2; ++complex64) {
      const pxp::MixedLines l = pxp::mixed_lines(n, complex64);
      const unsigned long long smem = pxp::mixed_lines_smem(p, l.lines, complex64);
      most = smem > most ? smem : most;
      if (l.threads % 32 || l.threads < 64 || l.lines < 1 || l.lines > 2 || smem > 227 * 1024) {
        std::printf("FAIL %d complex%d: %d threads, %d lines, %llu bytes\n", n, complex64 ? 64 : 128,
                    l.threads, l.lines, smem);
        return 1;
      }
    }
  }
  std::printf("%llu bytes\nOK\n", most);
  return 0;
}
