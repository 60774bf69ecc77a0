// The FP32 test by which the section kernel skips segments (hg_section.cu).
// Compiles as device code and as host C++, so that it can be tested on the CPU.
#pragma once

#include "hg_exact.cuh"

// a / b for 0 <= a <= b below 2^101 (two ulps)
HG_XHD float hgs_ratio(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fdividef(a, b);
#else
  return a / b;
#endif
}

// Whether a segment certainly has no crossing, from FP32 values of its own and
// its neighbours' ends (gp before, gn after; dp, d, dn the segments' lengths; a
// missing neighbour is the nearer end again, at no length).
//
// Linear: every point is a convex combination of the ends.  Cubic: on [0, 1]
// the Hermite cubic with end slopes m0, m1 is the Bezier curve with control
// values g0, g0 + m0/3, g1 - m1/3, g1 and lies in their convex hull; it also
// satisfies g(s) = g0 H00 + g1 H01 + m0 H10 + m1 H11 with H00, H01 >= 0,
// H00 + H01 = 1, |H10|, |H11| <= 4/27.  Where either keeps the curve on the
// side of the (same-signed) ends by more than 2^-17 (|g0| + |g1| + |gp| + |gn|
// + |m0| + |m1|), no evaluated point changes sign: the FP32 values carry at
// most 2^-20 of those terms (m0 = (g1 - gp) d / (dp + d), the ratio at most 1
// and off by 2^-21), an FP64 point a few 2^-53.  Ends outside (2^-100, 2^100)
// decide nothing (among them those whose product underflows, which without a
// direction is a reported crossing), nor do lengths of 2^100 or negative ones.
HG_XHD bool hgs_surely_clear(bool cubic, float gp, float g0, float g1, float gn, float dp, float d, float dn) {
  const float a0 = fabsf(g0), a1 = fabsf(g1), lo = fminf(a0, a1);
  if (!(a0 > 0x1p-100f && a1 > 0x1p-100f && a0 < 0x1p100f && a1 < 0x1p100f) || (g0 > 0.0f) != (g1 > 0.0f)) return false;
  if (!cubic) return true;
  if (!(fabsf(gp) < 0x1p100f && fabsf(gn) < 0x1p100f && d > 0x1p-100f && d < 0x1p100f && dp >= 0.0f && dp < 0x1p100f &&
        dn >= 0.0f && dn < 0x1p100f))
    return false;
  const float m0 = (g1 - gp) * hgs_ratio(d, dp + d), m1 = (gn - g0) * hgs_ratio(d, d + dn);
  const float am = fabsf(m0) + fabsf(m1);
  const float margin = 0x1p-17f * ((a0 + a1) + (fabsf(gp) + fabsf(gn)) + am);
  const float sg = g0 > 0.0f ? 1.0f : -1.0f;
  const bool hull = sg * (g0 + m0 * 0.33333334f) > margin && sg * (g1 - m1 * 0.33333334f) > margin && lo > margin;
  return hull || lo > 0.14814816f * am + margin;
}
