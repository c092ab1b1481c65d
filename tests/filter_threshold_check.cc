// Checks the filter kernels' threshold arithmetic (wmh_internal.h): the 16-bit
// difference never leaves 16 bits, it passes an entry exactly when byte < T, and
// an infinite weight passes for every byte at every threshold.  Prints "ok".
#include <climits>
#include <cstdio>

#include "wmh_internal.h"

int main() {
  int bad = 0;
  const int ms[] = {mhb::clamp_min(INT_MIN), -8192, -8191, -4096, -300, -1, 0, 1, 300, 8190, mhb::clamp_min(INT_MAX)};
  const int ls[] = {mhb::clamp_weight(INT_MIN), -2080, -1, 0, 1, 1775, 8191, 8192, mhb::clamp_weight(INT_MAX)};
  for (int m : ms) {
    if (mhb::clamp_min(m) != m) ++bad;
    // The kernel raises l so that T >= 1 (byte 0 always passes).
    const int least = 1 - 241 - m;
    for (int l0 : ls) {
      if (mhb::clamp_weight(l0) != l0) ++bad;
      const int l = l0 > least ? l0 : least;
      for (unsigned byte = 0; byte < 256; ++byte) {
        const unsigned d = mhb::filter_diff(byte, m, l);
        const bool passes = !(d & 0x8000u);
        if (d > 0xFFFFu || passes != (static_cast<int>(byte) < m + l + 241)) ++bad;
        if (l0 == mhb::clamp_weight(INT_MAX) && !passes) {
          if (byte == 255) printf("an infinite weight is skipped at m = %d\n", m);
          ++bad;
        }
      }
    }
  }
  if (bad == 0) puts("ok");
  return bad != 0;
}
