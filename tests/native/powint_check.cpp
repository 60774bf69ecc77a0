// Checks the integer-pipe powers (hg_powint.cuh), compiled as host C++, against
// quad-precision pow rounded once: the controller's three exponents on random
// errors over the whole range, every table entry's first and last significand,
// and significands next to a power of two.  A power whose `ok` is set must be
// the correctly rounded one.  The same for x^1.5 and x^2.5.  Prints
// "<powers> <wrong> <random powers> <of them ok> <random x^1.5, x^2.5> <of them ok>".
#include <stdio.h>
#include <stdlib.h>

#include <initializer_list>

#include "hg_powint.cuh"
#if defined(__aarch64__)
typedef long double q_t;
#define QPOW powl
#else
#include <quadmath.h>
typedef __float128 q_t;
#define QPOW powq
#endif

static uint64_t state = 1;
static uint64_t next64() {  // splitmix64
  uint64_t z = (state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
static long powers, wrong, random_powers, random_ok, roots, root_ok;
static double make(uint64_t bits) {
  double x;
  memcpy(&x, &bits, 8);
  return x;
}
// x^1.5 and x^2.5 with the FP32 estimate k ulps from the best
static void check_r2(uint64_t bits, int k) {
  const double x = make(bits);
  const double t = 1.0 / sqrt((double)hgx_sqrt_arg(x));
  float y = hgx_float(hgx_fbits((float)t) + (uint32_t)k);
  if (fabs(y / t - 1.0) > 1.2783e-7) y = (float)t;
  for (bool want25 : {false, true}) {
    bool ok;
    const double p = hgp_pow15_or_25(x, y, want25, ok);
    ++roots;
    root_ok += ok;
    if (ok && p != (double)QPOW((q_t)x, (q_t)(want25 ? 2.5 : 1.5))) ++wrong;
  }
}
static void check(uint64_t bits, bool random) {
  double x;
  memcpy(&x, &bits, 8);
  const double beta = 1.0 / 9.0, ys[3] = {-beta, 0.4 * beta, -0.125};
  const HgLog2 g = hgp_log2(x);
  for (double y : ys) {
    if (fabs(y * log(x)) > 85.0) continue;
    bool ok;
    const double p = hgp_exp(g, (uint64_t)(fabs(y) * 0x1p64), y < 0.0, ok);
    ++powers;
    if (random) ++random_powers, random_ok += ok;
    if (ok && p != (double)QPOW((q_t)x, (q_t)y)) ++wrong;
  }
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 100000;
  for (uint64_t j = 0; j < 1024; ++j)
    for (uint64_t e : {(uint64_t)1, (uint64_t)990, (uint64_t)1022, (uint64_t)1023, (uint64_t)1024, (uint64_t)2018}) {
      check((e << 52) | (j << 42), false);
      check((e << 52) | (j << 42) | ((1ull << 42) - 1), false);
    }
  for (long i = 0; i < n; ++i) {
    const uint64_t r = next64(), m = next64() >> 12;
    check(((1 + r % 2018) << 52) | m, true);
    check(((983 + r % 50) << 52) | m, true);
    check(((983 + r % 50) << 52) | ((r >> 40) & 1 ? (1ull << 52) - 1 - (m & 15) : (m & 15)), false);
  }
  long edges = 0, edge_ok = 0;
  for (long i = 0; i < n; ++i) {
    const uint64_t r = next64(), m = next64() >> 12;
    check_r2(((983 + r % 80) << 52) | m, (int)((r >> 32) % 5) - 2);
    edges -= roots, edge_ok -= root_ok;
    check_r2(((983 + r % 80) << 52) | ((r >> 40) & 1 ? (1ull << 52) - 1 - (m & 255) : (m & 255)), 0);
    edges += roots, edge_ok += root_ok;
  }
  roots -= edges, root_ok -= edge_ok;
  for (double x : {0.0, -1.0, 5e-324, 1e-40, 1e40, (double)INFINITY, (double)NAN})
    for (bool want25 : {false, true}) {
      bool ok;
      hgp_pow15_or_25(x, 1.0f, want25, ok);
      if (ok) ++wrong;
    }
  for (double x : {0.0, -1.0, 5e-324, 1e-310, (double)INFINITY, (double)NAN})
    if (hgp_log2(x).ok) ++wrong;
  printf("%ld %ld %ld %ld %ld %ld\n", powers, wrong, random_powers, random_ok, roots, root_ok);
  return 0;
}
