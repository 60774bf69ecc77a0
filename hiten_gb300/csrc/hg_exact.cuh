// Correctly rounded FP64 square roots and quotients on the FP32 and integer
// pipes.
//
// GB300's FP64 unit takes one lane operation per half clock and SM (a warp
// instruction holds it 16 cycles, and a warp alone waits 64 cycles for each),
// while the SM issues up to four FP32 / integer warp instructions per clock.
// A correctly rounded FP64 square root is eight FP64 instructions, a reciprocal
// five and a quotient three more (44 of a 6-dim right-hand side's 75 with two
// roots, two reciprocals and six quotients); here they take none.  The significands are exact integers, the estimates FP32:
//   * a 24-bit first estimate from the FP32 reciprocal (square root),
//   * two corrections, each the integer remainder of the estimate so far
//     (modulo 2^32 or 2^64: the remainders are small, so the low bits are all
//     of them) times the FP32 reciprocal,
//   * the second correction's distance from the rounding boundary.  The
//     estimate's error is bounded (derivations at the functions); when the
//     boundary is nearer than that, or an operand is outside the range
//     (2^-400, 2^400), `ok` is cleared and the caller takes the FP64
//     sequence for that value (less than one warp in fifty).
// A result with `ok` set is the correctly rounded one, so the bits are those
// of IEEE division and square root.
//
// The header compiles as device code and as host C++; the FP32 estimates are
// arguments, so that the bounds can be tested on the CPU with estimates of
// any admitted error.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#include "hg_crmath.cuh"
#define HG_XHD __host__ __device__ __forceinline__
#else
#define HG_XHD static inline
#endif

HG_XHD uint32_t hgx_hi(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)(b >> 32);
#endif
}
HG_XHD uint32_t hgx_lo(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2loint(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)b;
#endif
}
HG_XHD double hgx_make(uint32_t hi, uint32_t lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
HG_XHD uint32_t hgx_fbits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t b;
  memcpy(&b, &x, 4);
  return b;
#endif
}
HG_XHD float hgx_float(uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(b);
#else
  float x;
  memcpy(&x, &b, 4);
  return x;
#endif
}

// FP32 estimates (PTX: relative error at most 2^-23 and 2^-22.9).
HG_XHD float hgx_rcp_approx(float x) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.0f / x;
#endif
}
HG_XHD float hgx_rsqrt_approx(float x) {
#if defined(__CUDA_ARCH__)
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return (float)(1.0 / sqrt((double)x));
#endif
}

// fmaf(a, b, M) with M = 2^23 + m leaves a * b, rounded to the nearest
// integer, plus m in the low bits, for results in [2^23, 2^24).  The first
// corrections take m = HGX_M1, the second HGX_M2 = 2^22.
#define HGX_M1_BITS 0x4B2D3000u
#define HGX_M2_BITS 0x4B400000u
#define HGX_M1 11350016.0f
#define HGX_M2 12582912.0f
// The significand from the bits of its three parts: the first estimate f (an
// FP32 number with exponent -1 or 0: bits 0x3F000000 + 2^23 [exponent 0] +
// mantissa) at 2^29, the first correction at 2^10 and the second at 1.  M1 is
// the constant for which the three offsets add up to a multiple of 2^32,
// HGX_OFFSET 2^32, which the caller takes off the upper word.
#define HGX_OFFSET (0x12Du + 0x07E00000u)
// exponent fields of (2^-400, 2^400), as the doubled high word
#define HGX_EXP_LO ((1023u - 400u) << 21)
#define HGX_EXP_SPAN (800u << 21)

HG_XHD bool hgx_in_range(uint32_t hi) { return (hi << 1) - HGX_EXP_LO < HGX_EXP_SPAN; }
HG_XHD bool hgx_positive_in_range(uint32_t hi) { return hi - (HGX_EXP_LO >> 1) < (HGX_EXP_SPAN >> 1); }

HG_XHD uint32_t hgx_funnel_l(uint32_t lo, uint32_t hi, uint32_t sh) {  // sh modulo 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, sh);
#else
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << (sh & 31u)) >> 32);
#endif
}
HG_XHD int32_t hgx_mulhi(int32_t a, int32_t b) {
#if defined(__CUDA_ARCH__)
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
// a * b + addend (one multiply-add)
HG_XHD int64_t hgx_mad_wide(int32_t a, int32_t b, int64_t c) { return (int64_t)((uint64_t)((int64_t)a * b) + (uint64_t)c); }
HG_XHD uint64_t hgx_mad_wide_u(uint32_t a, uint32_t b, uint64_t c) { return (uint64_t)a * b + c; }
HG_XHD int64_t hgx_pack(uint32_t lo, uint32_t hi) { return (int64_t)(((uint64_t)hi << 32) | lo); }

// A positive divisor prepared for quotients.  D: its significand, 53 bits.
struct HgDen {
  int32_t h, l;  // -2^7 D = 2^32 h + l, l signed
  uint32_t ex;   // 1022 less the exponent field, in place, less HGX_OFFSET
  float y;       // (1 + e) 2^52 / D, |e| <= 2^-24 + 2^-40
  bool ok;
};

HG_XHD float hgx_den_arg(double d) {
  return hgx_float(0x3F800000u | (((hgx_hi(d) << 3) | (hgx_lo(d) >> 29)) & 0x7FFFFFu));
}
// y0: FP32 estimate of 1 / hgx_den_arg(d), relative error at most 2^-22.5;
// one Newton step that counts the 29 truncated bits leaves the rounding of y.
HG_XHD HgDen hgx_den(double d, float y0) {
  HgDen r;
  const uint32_t hi = hgx_hi(d), lo = hgx_lo(d);
  const uint64_t m = 0ull - (((uint64_t)((((hi & 0xFFFFFu) | 0x100000u) << 7) | (lo >> 25)) << 32) | (lo << 7));
  r.l = (int32_t)(uint32_t)m;
  r.h = (int32_t)((uint32_t)(m >> 32) + ((uint32_t)m >> 31));
  r.ex = (1022u << 20) - (hi & 0x7FF00000u) - HGX_OFFSET;
  r.ok = hgx_positive_in_range(hi);
  const float low = (float)(int32_t)(lo & 0x1FFFFFFFu);
  float e = fmaf(-hgx_den_arg(d), y0, 1.0f);
  e = fmaf(-low, y0 * 0x1p-52f, e);
  r.y = fmaf(y0, e, y0);
  return r;
}

// RN(n / d).  N: the significand; N' = N or 2N so that 1 <= N'/D < 2 and the
// quotient's significand is Q = RN(N' 2^52 / D).
//   qf = N/D from N's upper 32 bits: relative error at most 3 * 2^-24 + 2^-31.
//     N' = N when it is at least 1, else 2N; Q1 2^-23 is qf or 2 qf (24 bits),
//     |N'/D - Q1 2^-23| < 2^-21.4.  An estimate within 2^-20 of 1/2, 1 or 2,
//     where it could be on the wrong side, clears `ok`;
//   r1 = 2^30 N' - Q1 (2^7 D), below 2^61.6: its upper word r gives c1 =
//     RN(r y 2^-8) < 2^20.7, in units of 2^10 Q; what is left, in units of Q,
//     is at most 512 (rounding) + 2 * 98 (FP32 r and y) + 4 < 712;
//   r2 = 2^19 r1 - c1 (2^7 D): its upper word (off by at most two) gives c2 =
//     r2 y 2^-17 with an error of at most 2 * 712 * 2^-24 + 2^-16 < 2^-13.2,
//     so where it is more than 2^-13 from a half, c2 rounded is the nearest.
HG_XHD double hgx_quot(const HgDen& D, double n, bool& ok) {
  const uint32_t nhi = hgx_hi(n), nlo = hgx_lo(n);
  const float qf = (float)(hgx_funnel_l(nlo, nhi, 11) | 0x80000000u) * (D.y * 0x1p-31f);
  const uint32_t qb = hgx_fbits(qf);
  const int32_t Q1 = (int32_t)((qb & 0x7FFFFFu) | 0x800000u);
  // exponent of qf 127: N' = N, shift 30; 126: N' = 2N, shift 31
  const uint32_t sh = (qb ^ 0x800000u) >> 23;
  const uint32_t r1h = hgx_funnel_l(nlo, nhi, sh) + (uint32_t)Q1 * (uint32_t)D.h;
  const uint64_t r1 = (uint64_t)hgx_mad_wide(Q1, D.l, hgx_pack(hgx_funnel_l(0u, nlo, sh), r1h));
  const float f1 = (float)(int32_t)(uint32_t)(r1 >> 32);
  const uint32_t b1 = hgx_fbits(fmaf(f1, D.y * 0x1p-8f, HGX_M1));
  const int32_t c1 = (int32_t)(b1 - HGX_M1_BITS);
  const uint32_t r2 = hgx_funnel_l((uint32_t)r1, (uint32_t)(r1 >> 32), 19) + (uint32_t)hgx_mulhi(c1, D.l) +
                      (uint32_t)c1 * (uint32_t)D.h;
  const float f2 = (float)(int32_t)r2;
  const float yk = D.y * 0x1p-17f;
  const float v = fmaf(f2, yk, HGX_M2);
  const float fr = fmaf(f2, yk, -(v - HGX_M2));
  const uint64_t Q = hgx_mad_wide_u(qb, 1u << 29, hgx_mad_wide_u(b1, 1024u, hgx_fbits(v)));
  ok = hgx_in_range(nhi) && ((qb + 8u) & 0x7FFFF0u) != 0u && fabsf(fr) < 0.49987793f;
  return hgx_make((uint32_t)(Q >> 32) + (nhi & 0xFFF00000u) + D.ex, (uint32_t)Q);
}

HG_XHD float hgx_sqrt_arg(double x) {
  // the significand's upper 24 bits in [1, 2), in [2, 4) for an even exponent field
  const uint32_t m = (hgx_hi(x) << 3) | (hgx_lo(x) >> 29);
  return hgx_float(((m & 0xFFFFFFu) ^ 0x800000u) + 0x3F800000u);
}

// RN(sqrt(x)); y: FP32 estimate of 1 / sqrt(hgx_sqrt_arg(x)), relative error
// at most 2^-22.9.  a: the significand, doubled for an even exponent field, so
// that the root's significand is S = RN(sqrt(a 2^52)), 2^52 <= S < 2^53.
//   S1 (24 bits): relative error at most 2^-22.9 (y) + 2^-24 (product) +
//     2^-24 (truncated argument), less towards 2^53: |S - S1 2^29| < 2^30.7;
//   r1 = a - 64 S1^2, below 2^32.7; r1 / 8 and r1 modulo 2^32 are 32-bit
//     words.  c1 = RN(r1 y 2^-11), in units of 2^10 S; what is left, in units
//     of S, is at most 512 (rounding) + 215 (y) + 100 (FP32 r1) + 154 (the
//     correction's square) + 4 < 990;
//   r2 = a 2^32 - (S1 2^19 + c1)^2 = 2^32 r1 - 2^20 S1 c1 - c1^2, below
//     2^44.5: / 2^14 it is a 32-bit word and an FP32 term, c2 = r2 y 2^-33
//     with an error of at most 990 * 2^-22.9 (y) + 2.1e-4 (FP32 sums) <
//     3.4e-4, so where it is more than 4e-4 from a half, c2 rounded is the
//     nearest.
// S_raw: S + 2^32 HGX_OFFSET; fr: sqrt(a 2^52) - S, off by at most 3.4e-4.
HG_XHD void hgx_sqrt_parts(double x, float y, uint64_t& S_raw, float& fr) {
  const uint32_t hi = hgx_hi(x), lo = hgx_lo(x);
  const uint32_t sh = (hi >> 20) & 1u;  // 1: a is the significand, 0: twice it
  const uint32_t alo = lo << (1u - sh);
  const uint32_t a3 = hgx_funnel_l(lo, hi, 30u - sh);  // low word of a / 8
  const uint32_t sb = hgx_fbits(hgx_sqrt_arg(x) * y);
  const uint32_t S1 = sb - 0x3F000000u;
  const uint32_t q = S1 * S1;
  const float f1 = (float)(int32_t)(a3 - q * 8u);
  const float v1 = fmaf(f1, y * 0x1p-8f, HGX_M1);
  const uint32_t b1 = hgx_fbits(v1);
  const uint32_t c1 = b1 - HGX_M1_BITS;
  const float c1f = v1 - HGX_M1;
  const int32_t ri = (int32_t)(((alo - q * 64u) << 18) - S1 * (c1 << 6));
  const float f2 = fmaf(c1f, c1f * -0x1p-14f, (float)ri);
  const float yk = y * 0x1p-19f;
  const float v = fmaf(f2, yk, HGX_M2);
  fr = fmaf(f2, yk, -(v - HGX_M2));
  S_raw = hgx_mad_wide_u(sb, 1u << 29, hgx_mad_wide_u(b1, 1024u, hgx_fbits(v)));
}
HG_XHD double hgx_sqrt(double x, float y, bool& ok) {
  uint64_t S;
  float fr;
  hgx_sqrt_parts(x, y, S, fr);
  const uint32_t hi = hgx_hi(x);
  ok = hgx_positive_in_range(hi) && fabsf(fr) < 0.4996f;
  const uint32_t ex = ((hi + (1021u << 20)) >> 1) & 0x7FF00000u;
  return hgx_make((uint32_t)(S >> 32) + (ex - HGX_OFFSET), (uint32_t)S);
}

#if defined(__CUDACC__)
// Device forms, with the FP64 sequences behind them for the values whose `ok`
// is cleared (branches after the whole group's results, so that the group's
// instruction streams interleave).
__device__ __forceinline__ HgDen hg_den(double d) { return hgx_den(d, hgx_rcp_approx(hgx_den_arg(d))); }

// RN(sqrt(x)).  The FP64 root behind it is volatile: the compiler takes the
// root of a plain sqrt() on every path and selects, which puts its eight FP64
// instructions back.
__device__ __forceinline__ double hg_sqrt(double x) {
  bool ok;
  double s = hgx_sqrt(x, hgx_rsqrt_approx(hgx_sqrt_arg(x)), ok);
  if (!ok) asm volatile("sqrt.rn.f64 %0, %1;" : "=d"(s) : "d"(x));
  return s;
}

// n / d
__device__ __forceinline__ double hg_div(double n, double d) {
  const HgDen D = hg_den(d);
  bool ok;
  double q = hgx_quot(D, n, ok);
  if (!(ok && D.ok)) asm volatile("div.rn.f64 %0, %1, %2;" : "=d"(q) : "d"(n), "d"(d));
  return q;
}

// q[i] = RN(n[i] / d): the values of hg_div_rn(n[i], d, hg_rcp_rn(d))
template <int K>
__device__ __forceinline__ void hg_quotients(const double (&n)[K], double d, double (&q)[K]) {
  const HgDen D = hg_den(d);
  bool ok[K], all = D.ok;
#pragma unroll
  for (int i = 0; i < K; ++i) {
    q[i] = hgx_quot(D, n[i], ok[i]);
    all = all && ok[i];
  }
  if (!all) {
    // zero numerators (a planar problem's z) need no FP64 sequence: +0
    bool need = !D.ok;
#pragma unroll
    for (int i = 0; i < K; ++i) {
      if (hg_eq0(n[i]))
        q[i] = 0.0;
      else
        need = need || !ok[i];
    }
    if (need) {
      const double rd = hg_rcp_rn(d);
#pragma unroll
      for (int i = 0; i < K; ++i) q[i] = hg_div_rn(n[i], d, rd);
    }
  }
}
#endif
