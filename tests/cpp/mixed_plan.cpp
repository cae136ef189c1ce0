// The mixed-radix plan of every length it takes, checked without a GPU: the
// radices multiply to n and are ones the kernels have, every pass's index
// division is exact, the table holds what the passes read, and two buffers
// and the table fit shared memory; lengths it must not take are refused.
#include <cstdio>

#include "../../paxpro_b200/csrc/mixed_plan.h"

static int fail(const char *what, int n) {
  std::printf("FAIL %s at %d\n", what, n);
  return 1;
}

int main() {
  int taken = 0;
  for (int n = 1; n <= 8192; ++n) {
    pxp::MixedPlan p;
    const bool ok = pxp::mixed_plan(n, &p);
    int rest = n;
    for (int q = 2; q <= 31; ++q)
      while (rest % q == 0) rest /= q;
    const bool want = n >= 2 && n <= 4096 && (n & (n - 1)) && rest == 1;
    if (ok != want) return fail("choice", n);
    if (!ok) continue;
    ++taken;
    long long prod = 1;
    int table = n - 1, last = 0;
    bool big = false;
    for (int i = 0; i < p.passes; ++i) {
      const auto &q = p.pass[i];
      switch (q.radix) {
        case 2: case 3: case 4: case 5: case 7: case 8: case 9: case 11: case 13:
        case 17: case 19: case 23: case 29: case 31: break;
        default: return fail("radix", n);
      }
      big = big || q.radix > 13;
      if (q.nb * q.radix != n) return fail("butterflies", n);
      for (int b = 0; b < q.nb && prod > 1; ++b)
        if ((int)(((unsigned long long)b * q.magic) >> 32) != b / (int)prod) return fail("division", n);
      if (q.radix > 9) {
        if (q.radix != last) {
          if (q.rot != table) return fail("factors", n);
          table += (q.radix / 2) * (q.radix / 2);
        } else if (q.rot != p.pass[i - 1].rot) {
          return fail("repeated factors", n);
        }
      }
      last = q.radix;
      prod *= q.radix;
    }
    if (prod != n || p.table != table || p.big != big) return fail("plan", n);
    if (2 * 16 * n + 16 * p.table > 225 * 1024) return fail("shared memory", n);
  }
  std::printf("%d lengths\nOK\n", taken);
  return 0;
}
