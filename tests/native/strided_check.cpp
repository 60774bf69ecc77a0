// Strided / blocks_of at the ends of their range.  Prints the number of loops
// checked and of wrong ones.
#include "hg_strided.cuh"

#include <initializer_list>
#include <limits.h>
#include <stdio.h>

int main() {
  const long long counts[] = {0, 1, 255, 256, 311295, 311296, 311297, INT_MAX - 311297ll, INT_MAX - 311296ll,
                              INT_MAX - 128ll, INT_MAX - 127ll, INT_MAX - 1ll, INT_MAX};
  const long long steps[] = {1 << 20, 311296, 77824};
  int loops = 0, wrong = 0;
  for (long long n : counts) {
    for (int block : {128, 256}) {
      const unsigned b = blocks_of(n, block);
      ++loops;
      if ((long long)b * block < n || (long long)b * block >= n + block) ++wrong;
    }
    for (long long step : steps)
      for (long long first : {0ll, 1ll, 127ll, step / 2, step - 1}) {
        long long want = first, seen = 0;
        bool ok = true;
        for (const int i : Strided{first, step, n}) {
          ok = ok && i == want && want < n;
          want += step;
          if (++seen > n) break;  // (a loop that does not end)
        }
        ok = ok && seen == (first < n ? (n - first + step - 1) / step : 0);
        ++loops;
        if (!ok) ++wrong;
      }
  }
  printf("%d %d\n", loops, wrong);
  return 0;
}
