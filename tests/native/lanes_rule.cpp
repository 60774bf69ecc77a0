// Prints hg_internal's layout choices: for every n on the command line lanes_d6 and
// lanes_d42_free of n trajectories on `sms` multiprocessors.
#include "hg_internal.h"

#include <stdio.h>
#include <stdlib.h>

int main(int argc, char** argv) {
  const int sms = atoi(argv[1]);
  const double cap = atof(argv[2]);
  for (int k = 3; k < argc; ++k) {
    const long long n = atoll(argv[k]);
    printf("%lld %d %d\n", n, hg_internal::lanes_d6(n, sms, cap), hg_internal::lanes_d42_free(n, sms, cap));
  }
  return 0;
}
