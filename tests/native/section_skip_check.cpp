// Checks the section kernel's FP32 segment skip (hg_section_skip.cuh), compiled
// as host C++: where it calls a segment clear, every sub-interval point of the
// reference's Hermite form in binary64 has the end values' sign.  Segments with
// neighbours at random, with slopes that bring the curve's lowest point near
// zero, with neighbours far beyond the ends, at scales over the FP32 range, and
// without a neighbour on either side.  Prints "<segments> <clear> <wrong>".
#include <stdio.h>
#include <stdlib.h>

#include "hg_section_skip.cuh"

static uint64_t state = 1;
static uint64_t next64() {  // splitmix64
  uint64_t z = (state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
static double uni(double a, double b) { return a + (b - a) * ((double)(next64() >> 11) * 0x1p-53); }
static double herm(double s, double y0, double y1, double dy0, double dy1, double dt) {
  const double om = 1.0 - s;
  const double h00 = (1.0 + 2.0 * s) * (om * om), h10 = s * (om * om), h01 = (s * s) * (3.0 - 2.0 * s),
               h11 = (s * s) * (s - 1.0);
  return ((h00 * y0 + (h10 * dy0) * dt) + h01 * y1) + (h11 * dy1) * dt;
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  long clear = 0, wrong = 0;
  for (long i = 0; i < n; ++i) {
    const double scale = ldexp(1.0, i % 7 == 0 ? (int)(next64() % 220) - 110 : (int)(next64() % 30) - 25);
    const double sign = next64() & 1 ? 1.0 : -1.0;
    const double g0 = sign * scale * uni(0.01, 1.0), g1 = sign * scale * uni(0.01, 1.0) * (i % 11 == 0 ? -1.0 : 1.0);
    const double d = ldexp(uni(0.5, 1.0), (int)(next64() % 40) - 30);
    double dp = d * uni(0.1, 3.0), dn = d * uni(0.1, 3.0);
    // slopes (times d): at random, or the basis bound or a control value just
    // met, a little inside and outside
    double m0, m1;
    const double lo = fmin(fabs(g0), fabs(g1)), f = 1.0 + uni(-1.0, 1.0) * ldexp(1.0, -(int)(next64() % 24));
    switch (i % 4) {
      case 0: m0 = -sign * lo * uni(0.0, 8.0), m1 = sign * lo * uni(0.0, 8.0); break;
      case 1: m0 = -sign * lo * 3.375 * f, m1 = -m0; break;
      case 2: m0 = -3.0 * g0 * f, m1 = 3.0 * g1 * f; break;
      default: m0 = scale * uni(-30.0, 30.0), m1 = scale * uni(-30.0, 30.0); break;
    }
    double gp = g1 - m0 * (dp + d) / d, gn = g0 + m1 * (d + dn) / d;
    const bool left = i % 13 != 0, right = i % 17 != 0;
    if (!left) gp = g0, dp = 0.0;
    if (!right) gn = g1, dn = 0.0;
    ++wrong;
    if (!hgs_surely_clear(true, (float)gp, (float)g0, (float)g1, (float)gn, (float)dp, (float)d, (float)dn)) {
      --wrong;
      continue;
    }
    ++clear;
    const double d0 = (g1 - gp) / (d + dp), d1 = (gn - g0) / (dn + d);
    bool ok = (g0 > 0.0) == (g1 > 0.0);
    for (int q = 0; q <= 51; ++q) {
      const double v = herm((double)q * (1.0 / 51.0), g0, g1, d0, d1, d);
      ok = ok && (g0 > 0.0 ? v > 0.0 : v < 0.0);
    }
    wrong -= ok;
    if (!hgs_surely_clear(false, 0.0f, (float)g0, (float)g1, 0.0f, 0.0f, (float)d, 0.0f)) ++wrong;
  }
  const float bad[] = {0.0f, -0.0f, INFINITY, -INFINITY, NAN, 1e-35f, 1e35f};
  for (float v : bad) {
    if (hgs_surely_clear(true, 1.0f, v, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f) || hgs_surely_clear(false, 1.0f, 1.0f, v, 1.0f, 1.0f, 1.0f, 1.0f) ||
        hgs_surely_clear(true, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, v, 1.0f))
      ++wrong;
    if (v != v || v > 1e34f || v < -1e34f)
      if (hgs_surely_clear(true, v, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f) || hgs_surely_clear(true, 1.0f, 1.0f, 1.0f, v, 1.0f, 1.0f, 1.0f) ||
          hgs_surely_clear(true, 1.0f, 1.0f, 1.0f, 1.0f, v, 1.0f, 1.0f) || hgs_surely_clear(true, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, v))
        ++wrong;
  }
  printf("%ld %ld %ld\n", n, clear, wrong);
  return 0;
}
