// Checks the wider form of x^1.5 and x^2.5 (hg_powint.cuh), compiled as host
// C++, against quad-precision products and roots rounded once: on values
// whose first form is undecided, on every sixteenth other one, on significands
// next to a power of two and of few bits (exact powers, ties), with FP32
// estimates of any admitted error.  Prints
// "<powers> <wrong> <undecided> <of them random>".
#include <math.h>
#include <stdio.h>

#include "hg_powint.cuh"
#if defined(__aarch64__)
typedef long double q_t;
#define QSQRT sqrtl
#else
#include <quadmath.h>
typedef __float128 q_t;
#define QSQRT sqrtq
#endif

static uint64_t state = 3;
static uint64_t next64() {  // splitmix64
  uint64_t z = (state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
static long powers, wrong, undecided;
static void check(uint64_t bits, bool all) {
  double x;
  memcpy(&x, &bits, 8);
  const double t = 1.0 / sqrt((double)hgx_sqrt_arg(x));
  float y = hgx_float(hgx_fbits((float)t) + (uint32_t)((int)(next64() % 3) - 1));
  if (fabs(y / t - 1.0) > 1.2783e-7) y = (float)t;
  for (int want25 = 0; want25 < 2; ++want25) {
    bool ok, okw;
    const double p = hgp_pow15_or_25(x, y, want25 != 0, ok);
    if (ok && !all) continue;
    const double w = hgp_pow15_or_25_wide(x, y, want25 != 0, okw);
    ++powers;
    if (!okw) {
      ++undecided;
      continue;
    }
    const q_t q = x;
    if (w != (double)(want25 ? q * q * QSQRT(q) : q * QSQRT(q)) || (ok && w != p)) ++wrong;
  }
}
int main() {
  for (long i = 0; i < 4000000; ++i) {
    const uint64_t span = i % 4 ? 199 : 6;  // |e| < 100
    const uint64_t e = 1023 - span / 2 + next64() % span;
    check(e << 52 | next64() >> 12, i % 16 == 0);
  }
  const long undecided_random = undecided;
  for (uint64_t e = 924; e < 1123; ++e)
    for (uint64_t k = 0; k < 64; ++k) {
      check(e << 52 | k, true);
      check((e << 52 | 0xFFFFFFFFFFFFFull) - k, true);
      check(e << 52 | k << 46, true);
    }
  printf("%ld %ld %ld %ld\n", powers, wrong, undecided, undecided_random);
  return wrong ? 1 : 0;
}
