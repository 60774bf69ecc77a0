// Checks the integer-pipe square root and quotient (hg_exact.cuh), compiled as
// host C++, against IEEE sqrt and division: random significands, significands
// next to a binade edge and quotients next to 1, exponents over the whole
// range, and FP32 estimates moved to the ends of their admitted error.  A
// result whose `ok` is set must be the IEEE one.  Prints
// "<samples> <wrong> <random quotients> <of them ok> <random roots> <of them ok>".
#include <stdio.h>
#include <stdlib.h>

#include "hg_exact.cuh"

static uint64_t state;
static uint64_t next64() {  // splitmix64
  uint64_t z = (state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
static uint64_t bits(double x) {
  uint64_t b;
  memcpy(&b, &x, 8);
  return b;
}
static double make(uint64_t mant, int e, unsigned sign) {
  const uint64_t b = ((uint64_t)sign << 63) | ((uint64_t)e << 52) | mant;
  double x;
  memcpy(&x, &b, 8);
  return x;
}
// the FP32 estimate of t moved by k ulps, where the error stays admitted
static float estimate(double t, int k, double limit) {
  const float y = hgx_float(hgx_fbits((float)t) + (uint32_t)k);
  return fabs((double)y / t - 1.0) <= limit ? y : (float)t;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  state = argc > 2 ? strtoull(argv[2], 0, 10) : 1;
  const uint64_t full = (1ull << 52) - 1;
  long wrong = 0, rq = 0, rqo = 0, rs = 0, rso = 0;
  for (long i = 0; i < n; ++i) {
    const uint64_t a = next64(), b = next64(), c = next64();
    uint64_t ma = a >> 12, mb = b >> 12;
    switch (i % 8) {
      case 1: ma = full - (a & 15); break;
      case 2: mb = full - (b & 15); break;
      case 3: ma = a & 15; break;
      case 4: mb = b & 15; break;
      case 5: ma = (mb + (a & 31) - 16) & full; break;
      case 6: ma = (mb + ((a & 31) - 16) * 0x8000000ull) & full; break;
      default: break;
    }
    const bool random = i % 8 == 0 || i % 8 == 7;
    // exponents over the accepted range, and (one in sixteen) beyond it
    const int span = (c & 15) == 0 ? 1021 : 399;
    const int ea = 1023 - span + (int)((c >> 8) % (2 * span)), eb = 1023 - span + (int)((c >> 24) % (2 * span));
    const double x = make(ma, ea, (unsigned)(c >> 5) & 1u), d = make(mb, eb, 0);
    const int k = (int)((c >> 40) % 5) - 2;
    const HgDen D = hgx_den(d, estimate(1.0 / (double)hgx_den_arg(d), k, 0x1p-22 * 0.70710678));
    bool ok;
    const double q = hgx_quot(D, x, ok);
    if (span == 399) {
      if (!D.ok) ++wrong;
      if (random) ++rq, rqo += ok;
    }
    if (ok && D.ok && bits(q) != bits(x / d)) ++wrong;
    const double s = hgx_sqrt(d, estimate(1.0 / sqrt((double)hgx_sqrt_arg(d)), k, 1.2783e-7), ok);
    if (random && span == 399) ++rs, rso += ok;
    if (ok && bits(s) != bits(sqrt(d))) ++wrong;
  }
  // values the functions must hand back
  const double bad[] = {0.0, -0.0, -1.0, 5e-324, 1e-310, INFINITY, -INFINITY, NAN, 1e200, 1e-200};
  for (double x : bad) {
    bool ok;
    hgx_sqrt(x, 1.0f, ok);
    if (ok) ++wrong;
    const HgDen D = hgx_den(x, 1.0f);
    if (D.ok) ++wrong;
    if (x != -1.0) {
      const HgDen one = hgx_den(1.5, hgx_rcp_approx(1.5f));
      hgx_quot(one, x, ok);
      if (ok) ++wrong;
    }
  }
  printf("%ld %ld %ld %ld %ld %ld\n", n, wrong, rq, rqo, rs, rso);
  return 0;
}
