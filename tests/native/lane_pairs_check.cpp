// Lane-paired blocks ([16 pairs][len][2], entry e of lane l at 2 (l / 2 len + e) + l % 2): the
// range asked for ahead of a task's G lanes holds every one of their values and, rounded
// outwards to 16 bytes, stays inside the block, for every lane, value size and length.
#include <cstdio>

#include "internal.h"

int main() {
  long ranges = 0;
  for (int wsize : {4, 8})
    for (int G : {1, 2, 4})
      for (long long m = 1; m <= 24; ++m)
        for (int lane = 0; lane < 32; lane += G) {
          const long long len = m * m;
          const long long a = mpf::pair_first(len, lane), b = a + mpf::pair_values(len, G);
          const long long lo = a * wsize / 16 * 16, hi = (b * wsize + 15) / 16 * 16;
          bool ok = lo >= 0 && hi <= 32 * len * wsize;
          for (int l = lane; l < lane + G; ++l)
            for (long long e : {0LL, len - 1}) {
              const long long at = (l >> 1) * len * 2 + (l & 1) + 2 * e;
              ok = ok && at >= a && at < b;
            }
          if (!ok) {
            std::printf("lane %d of %d, m %lld, %d bytes: [%lld, %lld) of %lld\n", lane, G, m, wsize, lo, hi,
                        32 * len * wsize);
            return 1;
          }
          ++ranges;
        }
  std::printf("ranges %ld\n", ranges);
  return 0;
}
