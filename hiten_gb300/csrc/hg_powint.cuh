// Correctly rounded powers on the integer pipes: x^y for the step-size
// controller's exponents, and x^1.5, x^2.5 of the variational equations.
//
// The controller.  hg_pow's logarithm and exponential (double-double, hg_crmath.cuh) are about
// 70 FP64 instructions each, 64 cycles apart for a warp alone: a tenth of a
// one-lane DOP853 step and a quarter of a six-lane one.  Here log2(x), its
// product with y and the power of two are 64-bit fixed-point numbers:
//   log2 x = e + L_j + log2(1 + z), 1 + z = m r_j exact (m the significand,
//     r_j a 17-bit reciprocal of its upper ten bits), 0 <= z < 2^-9.9, a
//     degree-5 polynomial; error below 6 units of 2^-64;
//   T = y (e + f): y is exact in 64 fractional bits, at most 1/8; error
//     below 0.5 + 6/8 < 1.3 units of 2^-64;
//   2^T = 2^n E_j 2^t, t < 2^-10, a degree-5 polynomial: R in [2^63, 2^64)
//     with an error below 0.5 (E_j) + 0.5 (last shift) + 1.3 ln 2 + 0.1 <
//     2.1 units.
// R's upper 53 bits, rounded, are the correctly rounded power unless R lies
// within those 2.1 units of a rounding boundary; then (one power in 340) `ok`
// is cleared and the caller takes the double-double form.
#pragma once

#include "hg_exact.cuh"
#include "hg_powint_tables.h"

#if defined(__CUDACC__)
__device__ static const uint32_t hg_d_pi_r[1024] = HG_PI_R_INIT;
__device__ static const unsigned long long hg_d_pi_l[1024] = HG_PI_L_INIT;
__device__ static const unsigned long long hg_d_pi_e[1024] = HG_PI_E_INIT;
#endif
#if defined(__CUDA_ARCH__)
#define HG_PI_TAB(name, i) __ldg(&hg_d_pi_##name[i])
#else
static const uint32_t hg_h_pi_r[1024] = HG_PI_R_INIT;
static const unsigned long long hg_h_pi_l[1024] = HG_PI_L_INIT;
static const unsigned long long hg_h_pi_e[1024] = HG_PI_E_INIT;
#define HG_PI_TAB(name, i) (hg_h_pi_##name[i])
#endif

HG_XHD uint32_t hgp_mulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
HG_XHD uint64_t hgp_mulhi64(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// log2(x) = (field - 1023) + f 2^-64 for normal x > 0 (`ok`).
struct HgLog2 {
  uint32_t field;
  uint64_t f;
  bool ok;
};

HG_XHD HgLog2 hgp_log2(double x) {
  HgLog2 r;
  const uint32_t hi = hgx_hi(x), lo = hgx_lo(x);
  r.ok = hi - 0x00100000u < 0x7FE00000u;  // positive, normal, finite
  r.field = hi >> 20;
  const uint32_t j = (hi >> 10) & 1023u;
  const uint32_t rj = HG_PI_TAB(r, j);
  // m r_j - 1 in units of 2^-68, shifted to units of 2^-73 (below 2^63.1)
  const uint64_t Z = ((uint64_t)lo * rj + ((uint64_t)(((hi & 0xFFFFFu) | 0x100000u) * rj) << 32)) << 5;
  const uint32_t zh = (uint32_t)(Z >> 32);
  const uint32_t t = HG_PI_A4 - hgp_mulhi(zh, HG_PI_A5);          // a4 - a5 z, 2^-24
  const uint32_t h = HG_PI_A3 - hgp_mulhi(zh, t);                 // a3 - z (..), 2^-33
  const uint64_t s = HG_PI_A2 - (((uint64_t)zh * h) >> 10);       // a2 - z (..), 2^-64
  const uint64_t w = HG_PI_A1 - (hgp_mulhi64(Z, s) >> 10);        // (a1 - z (..)) / 2, 2^-64
  r.f = HG_PI_TAB(l, j) + ((hgp_mulhi64(Z, w) + 128u) >> 8);
  return r;
}

// RN(x^y) or RN(x^-y) (`neg`) from log2 x; Y = y 2^64, 0 < y <= 1/8 a double.
HG_XHD double hgp_exp(const HgLog2& g, uint64_t Y, bool neg, bool& ok) {
  // T = y (field - 1023 + f): 32 integer and 64 fractional bits
  const uint64_t p0 = (uint64_t)g.field * (uint32_t)Y;
  const uint64_t p1 = (uint64_t)g.field * (uint32_t)(Y >> 32) + (p0 >> 32);
  const uint64_t k1 = 1023ull * (uint32_t)(Y >> 32) + ((1023ull * (uint32_t)Y) >> 32);
  const uint64_t a = (p1 << 32) | (uint32_t)p0, k = (k1 << 32) | (uint32_t)(1023u * (uint32_t)Y);
  const uint64_t b = hgp_mulhi64(g.f, Y);
  uint64_t T = a - k;
  uint32_t n = (uint32_t)(p1 >> 32) - (uint32_t)(k1 >> 32) - (a < k ? 1u : 0u);
  T += b;
  n += T < b ? 1u : 0u;
  if (neg) {  // 2^96 - T, the complement: one unit of 2^-64 less, on the side of the truncation
    T = ~T;
    n = ~n;
  }
  const uint32_t j = (uint32_t)(T >> 54);
  const uint64_t tq = T << 10;  // t, 2^-74
  const uint32_t th = (uint32_t)(tq >> 32);
  const uint32_t h3 = HG_PI_B3 + hgp_mulhi(th, HG_PI_B4 + hgp_mulhi(th, HG_PI_B5));  // b3 + t (b4 + t b5), 2^-36
  const uint64_t h2 = HG_PI_B2 + (((uint64_t)th * h3) >> 12);                         // 2^-66
  const uint64_t h1 = HG_PI_B1 + (hgp_mulhi64(tq, h2) >> 12);                         // 2^-64
  const uint64_t E = HG_PI_TAB(e, j);
  const uint64_t R = E + ((hgp_mulhi64(E, hgp_mulhi64(tq, h1)) + 512u) >> 10);        // 2^-63
  // upper 53 bits, rounded; the boundary (lower bits 1024) at least three
  // units away, and R not past 2^64 (t within an error of the next power)
  const uint64_t q = ((R >> 10) + 1u) >> 1;
  ok = g.ok && (((uint32_t)R + 1024u + 3u) & 2047u) >= 6u && (int64_t)R < 0;
  const uint64_t bits = q + ((uint64_t)(n + 1022u) << 52);
  return hgx_make((uint32_t)(bits >> 32), (uint32_t)bits);
}

// sqrt(x)'s significand s in 64 bits.
HG_XHD uint64_t hgp_root64(double x, float y) {
  uint64_t S_raw;
  float fr;
  hgx_sqrt_parts(x, y, S_raw, fr);
  return ((S_raw - ((uint64_t)HGX_OFFSET << 32)) << 11) +
         (uint64_t)(int64_t)(int32_t)(hgx_fbits(fmaf(fr, 2048.0f, HGX_M2)) - HGX_M2_BITS);
}
// x's significand in 64 bits
HG_XHD uint64_t hgp_significand64(double x) {
  const uint32_t hi = hgx_hi(x), lo = hgx_lo(x);
  return ((uint64_t)(((hi & 0xFFFFFu) | 0x100000u) << 11 | lo >> 21) << 32) | (lo << 11);
}
// The power from its significand R (upper 53 bits, rounded) and exponent: e +
// floor(e / 2), or 2 e + floor(e / 2), plus one for every product that reached
// 2 (sm, sr: those that did not).
HG_XHD double hgp_make_power(double x, uint64_t R, bool want25, uint32_t sm, uint32_t sr) {
  const int32_t e = (int32_t)(hgx_hi(x) >> 20) - 1023;
  const int32_t ex = e + (e >> 1) + (want25 ? e + 1 - (int32_t)sm : 0) + 1 - (int32_t)sr;
  const uint64_t q = ((R >> 10) + 1u) >> 1;
  const uint64_t bits = q + ((uint64_t)(uint32_t)(ex + 1022) << 52);
  return hgx_make((uint32_t)(bits >> 32), (uint32_t)bits);
}
// |e| < 100: the powers stay far from the ends of the range
HG_XHD bool hgp_power_range(double x) { return (hgx_hi(x) - (923u << 20)) < (200u << 20); }

// RN(x^1.5), or RN(x^2.5) when want25; y as for hgx_sqrt.  With x = m 2^e and
// sqrt(x) = s 2^k (1 <= m, s < 2), the significand is that of m s or m^2 s:
//   W: m in 64 bits (exact), or m^2's upper 64 (off by at most 1, centred);
//   S: s in 64 bits from the root's 53 and its remainder (off by at most
//     2048 * 3.4e-4 + 0.5 < 1.2);
//   R = W S / 2^64 normalised to [2^63, 2^64): off by at most 2 (1.2 + 0.5) =
//     3.4 units (x^1.5), 2 (1.2 + 1 + 0.5) = 5.4 (x^2.5).
// Closer than that to a rounding boundary (one value in 256 and in 170) `ok`
// is cleared.
HG_XHD double hgp_pow15_or_25(double x, float y, bool want25, bool& ok) {
  const uint64_t S = hgp_root64(x, y), m = hgp_significand64(x);
  uint64_t mm = hgp_mulhi64(m, m);
  const uint32_t sm = (uint32_t)(~mm >> 63);  // m^2 < 2
  mm = (mm << sm) + sm;
  const uint64_t W = want25 ? mm : m;
  uint64_t R = hgp_mulhi64(W, S);
  const uint32_t sr = (uint32_t)(~R >> 63);
  R = (R << sr) + sr;
  const uint32_t w = want25 ? 6u : 4u;
  ok = hgp_power_range(x) && (((uint32_t)R + 1024u + w) & 2047u) >= 2u * w;
  return hgp_make_power(x, R, want25, sm, sr);
}

// The same power for an `x` whose `ok` was cleared, with 30 more bits of the
// root: r = s^2 - S^2, exact modulo 2^128 and below 2^66, gives the root's
// next correction r / (2 S), an integer d in units of 2^-93, off by at most
// 1.2 * 2^30 * 2^-22.2 (y and two FP32 roundings) + 2 + 0.5 < 320.  The product
// with m (exact) or m^2 (106 bits, exact) in 128 bits is then off by less than
// 2 (320 * 2^34 + 3) = 2^43.4 units of its last bit, 2^-20.6 of R's.  `ok`
// stays cleared only within 2^-20 of a boundary.  A warp of five 42-dim
// trajectories takes twenty powers a right-hand side, so one right-hand side in
// ten came to the double-double form's forty FP64 instructions; with this form
// in between: fixed RK8 of 1024 states, 3000 steps, 98.7 -> 97.0 ms; 97
// monodromy matrices 2.76 -> 2.72 ms.
HG_XHD double hgp_pow15_or_25_wide(double x, float y, bool want25, bool& ok) {
  typedef unsigned __int128 u128;
  const uint64_t S = hgp_root64(x, y), m = hgp_significand64(x);
  const uint32_t odd = ~(hgx_hi(x) >> 20) & 1u;  // s^2 is m, or 2 m for an odd exponent
  const u128 r = ((u128)m << (63u + odd)) - (u128)S * S;
  const float rf = (float)(int32_t)(uint32_t)(uint64_t)(r >> 35);
  const int64_t d = (int64_t)rintf(rf * (2.0f * y));
  const u128 root = ((u128)S << 64) + (u128)((__int128)d << 34);
  const uint64_t Sh = (uint64_t)(root >> 64), Sl = (uint64_t)root;
  u128 W = (u128)m << 64;
  uint32_t sm = 0u;
  if (want25) {
    W = (u128)m * m;
    sm = (uint32_t)(~(uint64_t)(W >> 64) >> 63);
    W <<= sm;
  }
  const uint64_t Wh = (uint64_t)(W >> 64), Wl = (uint64_t)W;
  u128 P = (u128)Wh * Sh + hgp_mulhi64(Wl, Sh) + hgp_mulhi64(Wh, Sl);
  const uint32_t sr = (uint32_t)(~(uint64_t)(P >> 64) >> 63);
  P <<= sr;
  const uint64_t R = (uint64_t)(P >> 64);
  const uint64_t low = ((R & 2047u) << 32) | (uint32_t)((uint64_t)P >> 32);  // in units of 2^-32 of R's
  ok = hgp_power_range(x) && low - (1024ull << 32) + 4096u >= 8192u;
  return hgp_make_power(x, R, want25, sm, sr);
}

#if defined(__CUDACC__)
// x^1.5 or x^2.5, with the wider root and the double-double form behind it
__device__ __forceinline__ double hg_power_of_r2(double x, bool want25) {
  bool ok;
  const float y = hgx_rsqrt_approx(hgx_sqrt_arg(x));
  double p = hgp_pow15_or_25(x, y, want25, ok);
  if (!ok) {
    p = hgp_pow15_or_25_wide(x, y, want25, ok);
    if (!ok) p = hg_pow15_or_25(x, want25);
  }
  return p;
}
#endif
