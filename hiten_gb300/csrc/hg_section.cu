// Section-crossing detection on sampled trajectories (the synodic Poincare
// map), restating poincare/synodic/backend.py:458-659
// (_detect_with_segment_refine) and :382-455 (_order_and_dedup_hits) for an
// axis-aligned plane g = y[axis] - offset (SynodicMapConfig's section_axis /
// section_offset), linear sub-segment interpolation (the reference's
// default, see backend.py:762) or cubic Hermite with Newton refinement.
//
// A warp walks the segments of its 32 trajectories (one per lane) in lock
// step.  The reference scans every segment in (segment_refine + 1)
// sub-intervals; a segment that cannot hold a crossing is skipped by bounds
// that leave every evaluated point's sign certain, the scan of each remaining
// one is shared by the warp's lanes, and the crossings wait in a queue per lane
// until the lanes refine one each side by side.  Candidates leave a lane's
// queue in segment order, which is the reference's stable ordering, and are
// deduplicated against the last accepted hit as they stream out.
//
// What bounds it: a warp's FP64 chains, so what the scan does is kept small -- FP32
// bounds for the skip, the Hermite basis at the scan's points formed once per
// warp, every point evaluated once and handed to its neighbour -- and the
// chains of the refinements, which ran one lane at a time before they were
// queued.  20011 trajectories x 300 segments, cubic: 4.94 -> 0.70 ms (47 % of the
// FP64 unit on 3.9 warps an SM; the same launch takes 0.69 to 1.26 ms from process
// to process, by where its blocks land).
#include <cuda_runtime.h>
#include <math.h>

#include "hg_exact.cuh"
#include "hg_fp64_ops.cuh"
#include "hg_section_skip.cuh"
#include "hitengpu.h"

namespace {

struct SecParams {
  int N, m;
  const double* samples;  // [m][6][ld]
  long long ld;
  const double* times;    // [m][ld] (times_ld = ld) or [m] shared (times_ld = 0)
  long long times_ld;
  int axis;
  double offset;
  int direction;  // -1, 0 (any), +1
  int pu, pv;     // plane coordinates (projection) indices
  int segment_refine;
  int cubic;
  int newton_max_iter;
  double tol_on_surface, dedup_time_tol, dedup_point_tol;
  int max_hits;
  double* hit_t;  // [max_hits][ld]
  double* hit_y;  // [max_hits][6][ld]
  int* n_hits;    // stored hits
  int* n_found;   // accepted hits, including those beyond max_hits
};

__device__ __forceinline__ double smp(const SecParams& p, int q, int c, int i) {
  return p.samples[((long long)q * 6 + c) * p.ld + i];
}
__device__ __forceinline__ double tim(const SecParams& p, int q, int i) {
  return p.times_ld ? p.times[(long long)q * p.times_ld + i] : p.times[q];
}

// poincare/utils.py:53-147 (_hermite_scalar, _hermite_der: squares as x*x,
// the derivative is dH/ds), left-to-right association as written there.
__device__ __forceinline__ double hermite_scalar(double s, double y0, double y1, double dy0, double dy1, double dt) {
  const double om = 1.0 - s;
  const double h00 = (1.0 + 2.0 * s) * (om * om);
  const double h10 = s * (om * om);
  const double h01 = (s * s) * (3.0 - 2.0 * s);
  const double h11 = (s * s) * (s - 1.0);
  return ((h00 * y0 + (h10 * dy0) * dt) + h01 * y1) + (h11 * dy1) * dt;
}
__device__ __forceinline__ double hermite_der(double s, double y0, double y1, double dy0, double dy1, double dt) {
  const double om = 1.0 - s;
  const double dh00 = ((6.0 * s) * (s - 1.0) + (om * om) * 2.0) - (2.0 * om) * (1.0 + 2.0 * s);
  const double dh10 = om * om + s * (2.0 * (s - 1.0));
  const double dh01 = (6.0 * s) * om - (2.0 * s) * (3.0 - 2.0 * s);
  const double dh11 = (2.0 * s) * (s - 1.0) + s * s;
  return ((dh00 * y0 + (dh10 * dy0) * dt) + dh01 * y1) + (dh11 * dy1) * dt;
}

struct Emitter {
  const SecParams& p;
  int i;
  int stored = 0, found = 0;
  bool have = false;
  double pt = 0.0, pu = 0.0, pvv = 0.0;
  bool full = false;
  __device__ Emitter(const SecParams& pp, int ii) : p(pp), i(ii) {}
  // _order_and_dedup_hits: skip near-duplicates of the last accepted hit
  __device__ void offer(double th, const double (&x)[6]) {
    if (full) return;
    double u = x[0], v = x[0];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      if (c == p.pu) u = x[c];
      if (c == p.pv) v = x[c];
    }
    if (have) {
      if (fabs(th - pt) <= p.dedup_time_tol) return;
      const double du = u - pu, dv = v - pvv;
      if ((du * du + dv * dv) <= (p.dedup_point_tol * p.dedup_point_tol)) return;
    }
    have = true;
    pt = th;
    pu = u;
    pvv = v;
    ++found;
    if (stored < p.max_hits) {
      p.hit_t[(long long)stored * p.ld + i] = th;
#pragma unroll
      for (int c = 0; c < 6; ++c) p.hit_y[((long long)stored * 6 + c) * p.ld + i] = x[c];
      ++stored;
      if (stored >= p.max_hits) full = true;  // max_hits_per_traj cap (backend.py:451-452)
    }
  }
};

// One segment's scan: end values, end slopes (cubic) and length.
struct SegCtx {
  double gk, gk1, d0, d1, dt;
  bool cub;
};

// The segment k of trajectory i, as the reference forms it.
__device__ __forceinline__ SegCtx seg_ctx(const SecParams& p, int i, int k) {
  SegCtx c{smp(p, k, p.axis, i) - p.offset, smp(p, k + 1, p.axis, i) - p.offset, 0.0, 0.0, 0.0, false};
  const double tk = tim(p, k, i), tk1 = tim(p, k + 1, i);
  c.dt = tk1 - tk;
  c.cub = p.cubic && c.dt > 0.0;
  if (c.cub) {
    const bool left = k - 1 >= 0, right = k + 2 < p.m;
    const double ga = left ? smp(p, k - 1, p.axis, i) - p.offset : c.gk, ta = left ? tim(p, k - 1, i) : tk;
    const double gb = right ? smp(p, k + 2, p.axis, i) - p.offset : c.gk1, tb = right ? tim(p, k + 2, i) : tk1;
    c.d0 = hg_div(c.gk1 - ga, tk1 - ta);
    c.d1 = hg_div(gb - c.gk, tb - tk);
  }
  return c;
}

// The Hermite basis (cubic) or the linear weights at s, the products of
// hermite_scalar and of (1 - s) g0 + s g1 that depend on s alone.
struct Basis {
  double h00, h10, h01, h11, om;
  __device__ __forceinline__ explicit Basis(double s) {
    om = 1.0 - s;
    h00 = (1.0 + 2.0 * s) * (om * om);
    h10 = s * (om * om);
    h01 = (s * s) * (3.0 - 2.0 * s);
    h11 = (s * s) * (s - 1.0);
  }
  __device__ __forceinline__ double at(const SegCtx& c, double s) const {
    return c.cub ? ((h00 * c.gk + (h10 * c.d0) * c.dt) + h01 * c.gk1) + (h11 * c.d1) * c.dt : om * c.gk + s * c.gk1;
  }
};

__device__ __forceinline__ SegCtx from_lane(bool cubic, const SegCtx& c, int j) {
  SegCtx r{0.0, 0.0, 0.0, 0.0, 0.0, false};
  r.gk = __shfl_sync(0xFFFFFFFFu, c.gk, j);
  r.gk1 = __shfl_sync(0xFFFFFFFFu, c.gk1, j);
  if (cubic) {
    r.d0 = __shfl_sync(0xFFFFFFFFu, c.d0, j);
    r.d1 = __shfl_sync(0xFFFFFFFFu, c.d1, j);
    r.dt = __shfl_sync(0xFFFFFFFFu, c.dt, j);
    r.cub = __shfl_sync(0xFFFFFFFFu, (int)c.cub, j) != 0;
  }
  return r;
}

// Value of g at sub-interval point s of a segment: the cubic Hermite or the
// linear interpolant, as the reference evaluates it.
__device__ __forceinline__ double seg_point(const SegCtx& c, double s) {
  return c.cub ? hermite_scalar(s, c.gk, c.gk1, c.d0, c.d1, c.dt) : (1.0 - s) * c.gk + s * c.gk1;
}

__device__ __forceinline__ bool sub_crosses(double g_lo, double g_hi, int direction) {
  if (direction == 0) return (g_lo * g_hi <= 0.0) && (g_lo != g_hi);
  if (direction == 1) return hg_lt0(g_lo) && (hg_gt0(g_hi) || hg_eq0(g_hi));
  return hg_gt0(g_lo) && (hg_lt0(g_hi) || hg_eq0(g_hi));
}

// One warp a block: warps differ in their candidates, and a block of several
// holds its place until the slowest is done (cubic, us, blocks of 128 / 64 / 32
// in one process:
// 500 x 301 samples 657 / 619 / 593, 20011 x 301 918 / 803 / 738, 65536 x 301
// 1703 / 1412 / 1316).
constexpr int kSecBlock = 32;
constexpr int kSecQueue = 8;   // crossings a lane holds back
constexpr int kSecBatch = 8;   // samples loaded ahead

// Refine crossing mm of segment k (mm < 0: the segment's on-surface left end).
__device__ __noinline__ void emit_crossing(const SecParams& p, Emitter& em, int i, int k, int mm, double step) {
  double x[6];
  if (mm < 0) {
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) x[cc] = smp(p, k, cc, i);
    em.offer(tim(p, k, i), x);
    return;
  }
  const SegCtx c = seg_ctx(p, i, k);
  const double tk = tim(p, k, i), tk1 = tim(p, k + 1, i);
  const double s_lo = (double)mm * step;
  const double s_hi = (double)(mm + 1) * step;
  const double g_lo = seg_point(c, s_lo);
  const double g_hi = seg_point(c, s_hi);
  double s_star;
  if (g_lo == g_hi) {
    s_star = 0.5 * (s_lo + s_hi);
  } else {
    double a = hg_div(g_lo, g_lo - g_hi);
    a = fmin(1.0, fmax(0.0, a));
    s_star = s_lo + a * (s_hi - s_lo);
  }
  if (c.cub) {
    for (int it = 0; it < p.newton_max_iter; ++it) {
      const double f = hermite_scalar(s_star, c.gk, c.gk1, c.d0, c.d1, c.dt);
      const double df = hermite_der(s_star, c.gk, c.gk1, c.d0, c.d1, c.dt);
      if (df == 0.0) break;
      s_star -= hg_div(f, df);
      if (s_star < s_lo) {
        s_star = s_lo;
        break;
      }
      if (s_star > s_hi) {
        s_star = s_hi;
        break;
      }
    }
  }
  const double th = (1.0 - s_star) * tk + s_star * tk1;
  if (c.cub && k - 1 >= 0 && k + 2 < p.m) {
    const double tm1 = tim(p, k - 1, i), tp2 = tim(p, k + 2, i);
    const Basis b(s_star);
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) {
      const double x0 = smp(p, k, cc, i), x1 = smp(p, k + 1, cc, i);
      const double dxdt0 = hg_div(x1 - smp(p, k - 1, cc, i), tk1 - tm1);
      const double dxdt1 = hg_div(smp(p, k + 2, cc, i) - x0, tp2 - tk);
      x[cc] = ((b.h00 * x0 + (b.h10 * dxdt0) * c.dt) + b.h01 * x1) + (b.h11 * dxdt1) * c.dt;
    }
  } else {
#pragma unroll
    for (int cc = 0; cc < 6; ++cc) {
      const double a0 = smp(p, k, cc, i);
      x[cc] = a0 + s_star * (smp(p, k + 1, cc, i) - a0);
    }
  }
  em.offer(th, x);
}

__global__ void __launch_bounds__(kSecBlock) section_kernel(SecParams p) {
  __shared__ int q_seg[kSecQueue][kSecBlock], q_sub[kSecQueue][kSecBlock];
  __shared__ double s_g[2 * kSecBatch][kSecBlock], s_t[2 * kSecBatch][kSecBlock];
  const int tx = threadIdx.x;
  const int i = blockIdx.x * kSecBlock + tx;
  const int lane = tx & 31;
  const bool valid = i < p.N;
  const int ii = valid ? i : p.N - 1;
  Emitter em(p, ii);
  const int N = p.m;
  const int r = p.segment_refine;
  const double step = 1.0 / (double)(r + 1);
  const bool dir_any = p.direction == 0;
  // sub-intervals the reference scans: mm = 0 .. n_sub - 1 (it stops at the
  // first whose upper end exceeds 1 + 1e-15)
  int n_sub = 0;
  while (n_sub <= r && !((double)(n_sub + 1) * step > 1.0 + 1e-15)) ++n_sub;
  const int n_chunks = (n_sub + 31) / 32;
  // scan points of this lane in the first two chunks (the default 50-fold
  // refinement has 52 points)
  const double sa = (double)lane * step, sb = (double)(32 + lane) * step;
  const Basis ba(sa), bb(sb);

  int queued = 0;
  // every lane refines its queued crossings, one each side by side
  auto flush = [&]() {
    for (int e = 0; __any_sync(0xFFFFFFFFu, e < queued); ++e)
      if (e < queued && !em.full) emit_crossing(p, em, ii, q_seg[e][tx], q_sub[e][tx], step);
    queued = 0;
  };
  // push crossing mm of segment k; whole warp (flushes when a queue is full)
  auto push = [&](bool has, int k, int mm) {
    if (__any_sync(0xFFFFFFFFu, has && queued == kSecQueue)) flush();
    if (has) {
      q_seg[queued][tx] = k;
      q_sub[queued][tx] = mm;
      ++queued;
    }
  };

  auto push_bits = [&](unsigned bits, int k, int first) {
    while (__any_sync(0xFFFFFFFFu, bits != 0)) {
      push(bits != 0, k, first + __ffs(bits) - 1);
      bits &= bits - 1;
    }
  };

  // sample q of the section function and its time, two batches in shared memory
  auto load = [&](int q0, double (&g)[kSecBatch], double (&t)[kSecBatch]) {
#pragma unroll
    for (int e = 0; e < kSecBatch; ++e) {
      const int q = q0 + e < N ? q0 + e : N - 1;
      g[e] = smp(p, q, p.axis, ii);
      t[e] = tim(p, q, ii);
    }
  };
  auto store = [&](int q0, const double (&g)[kSecBatch], const double (&t)[kSecBatch]) {
#pragma unroll
    for (int e = 0; e < kSecBatch; ++e) {
      s_g[(q0 + e) % (2 * kSecBatch)][tx] = g[e] - p.offset;
      s_t[(q0 + e) % (2 * kSecBatch)][tx] = t[e];
    }
  };
  if (N < 2) {
    if (valid) {
      p.n_hits[i] = 0;
      if (p.n_found) p.n_found[i] = 0;
    }
    return;
  }
  double lg[kSecBatch], lt[kSecBatch];
  load(0, lg, lt);
  store(0, lg, lt);
  load(kSecBatch, lg, lt);
  // values at k - 1, k, k + 1 (own registers) and k + 2 (read below)
  double g_prev = 0.0, gk = s_g[0][tx], gk1 = s_g[1][tx];
  double t_prev = 0.0, tk = s_t[0][tx], tk1 = s_t[1][tx];
  float d_prev = 0.0f;
  for (int k = 0; k + 1 < N; ++k) {
    // sample k + 2 is in the buffers: batch k / 8 (and the next one, stored
    // when sample k + 2 is its first)
    if ((k + 2) % kSecBatch == 0) {
      store(k + 2, lg, lt);
      load(k + 2 + kSecBatch, lg, lt);
    }
    const bool live = valid && !em.full;
    if (!__any_sync(0xFFFFFFFFu, live)) break;
    const bool more = k + 2 < N;
    const double gk2 = more ? s_g[(k + 2) % (2 * kSecBatch)][tx] : 0.0;
    const double tk2 = more ? s_t[(k + 2) % (2 * kSecBatch)][tx] : tk1;
    const float d = (float)(tk1 - tk), d_next = (float)(tk2 - tk1);
    const float f0 = (float)gk, f1 = (float)gk1;
    const bool near = hg_gt0(p.tol_on_surface) && hg_bits(fabs(gk)) < hg_bits(p.tol_on_surface);
    const bool cand = live && (near || !hgs_surely_clear(p.cubic != 0, k > 0 ? (float)g_prev : f0, f0, f1,
                                                     more ? (float)gk2 : f1, k > 0 ? d_prev : 0.0f, d,
                                                     more ? d_next : 0.0f));
    bool skip0 = false, left_hit = false;
    if (cand && near) {
      if (dir_any)
        left_hit = true;
      else if (p.direction == 1)
        left_hit = (gk1 >= 0.0) || (k - 1 >= 0 && g_prev <= 0.0);
      else
        left_hit = (gk1 <= 0.0) || (k - 1 >= 0 && g_prev >= 0.0);
      skip0 = left_hit;
    }
    if (__any_sync(0xFFFFFFFFu, cand)) {
      if (__any_sync(0xFFFFFFFFu, left_hit)) push(left_hit, k, -1);
      // where one crossing is wanted, one at the segment's start is it, and the
      // segment needs no scan (32 trajectories that start on the surface, 301
      // samples, cubic: 92 -> 52 us)
      const unsigned cmask = __ballot_sync(0xFFFFFFFFu, cand && !(left_hit && p.max_hits == 1));
      SegCtx c{gk, gk1, 0.0, 0.0, tk1 - tk, false};
      c.cub = p.cubic && c.dt > 0.0;
      if (cand && c.cub) {
        c.d0 = hg_div(gk1 - (k > 0 ? g_prev : gk), tk1 - (k > 0 ? t_prev : tk));
        c.d1 = hg_div((more ? gk2 : gk1) - gk, tk2 - tk);
      }
      // every candidate segment is scanned by the whole warp: lane L evaluates
      // points L and 32 + L (further chunks below) and takes the next lane's as
      // its upper end
      unsigned bits0 = 0, bits1 = 0;
      for (unsigned rest = cmask; rest; rest &= rest - 1) {
        const int j = __ffs(rest) - 1;
        const SegCtx cj = from_lane(p.cubic != 0, c, j);
        const bool sk = __shfl_sync(0xFFFFFFFFu, (int)skip0, j) != 0;
        const double va = ba.at(cj, sa);
        const double ua = __shfl_down_sync(0xFFFFFFFFu, va, 1);
        double vb = 0.0, ub = 0.0;
        if (n_sub >= 32) {
          vb = bb.at(cj, sb);
          ub = __shfl_down_sync(0xFFFFFFFFu, vb, 1);
          if (n_sub >= 64 && lane == 31) ub = seg_point(cj, 64.0 * step);
        }
        const double v32 = __shfl_sync(0xFFFFFFFFu, vb, 0);
        const bool xa = lane < n_sub && !(sk && lane == 0) && sub_crosses(va, lane == 31 ? v32 : ua, p.direction);
        const bool xb = 32 + lane < n_sub && sub_crosses(vb, ub, p.direction);
        const unsigned m0 = __ballot_sync(0xFFFFFFFFu, xa), m1 = __ballot_sync(0xFFFFFFFFu, xb);
        if (lane == j) {
          bits0 = m0;
          bits1 = m1;
        }
      }
      push_bits(bits0, k, 0);
      push_bits(bits1, k, 32);
      for (int ch = 2; ch < n_chunks; ++ch) {
        unsigned bits = 0;
        for (unsigned rest = cmask; rest; rest &= rest - 1) {
          const int j = __ffs(rest) - 1;
          const SegCtx cj = from_lane(p.cubic != 0, c, j);
          const int mm = 32 * ch + lane;
          const bool x = mm < n_sub && sub_crosses(seg_point(cj, (double)mm * step),
                                                   seg_point(cj, (double)(mm + 1) * step), p.direction);
          const unsigned m = __ballot_sync(0xFFFFFFFFu, x);
          if (lane == j) bits = m;
        }
        push_bits(bits, k, 32 * ch);
      }
      // a lane that may have reached the cap finds out before it scans on
      if (__any_sync(0xFFFFFFFFu, live && queued > 0 && em.stored + queued >= p.max_hits)) flush();
    }
    d_prev = d;
    t_prev = tk;
    g_prev = gk;
    gk = gk1;
    gk1 = gk2;
    tk = tk1;
    tk1 = tk2;
  }
  flush();
  if (valid) {
    p.n_hits[i] = em.stored;
    if (p.n_found) p.n_found[i] = em.found;
  }
}

// Manifold acceptance filters on sampled trajectories
// (types/services/manifold.py:412-432): minimum distances to the primaries
// (np.sqrt((x + mu)**2 + y**2 + z**2), numpy squares being x*x) and the
// maximum relative Jacobi-constant drift of common/energy.py:26-74
// (numba: squares x*x, **0.5 of a positive number = the correctly rounded
// square root).
//
// One thread per trajectory and chunk of samples; chunks so many that the
// device is full (a manifold has tens to thousands of trajectories of thousands
// of samples: one thread for all samples of each left 12 of 152 SMs busy and
// took 16.3 ms for 1600 x 4713, 0.48 ms here; 0.49 with plain products and
// sums).  Bound: the FP64 unit, 27 instructions a sample (0.33 ms); the two roots and quotients are on the integer pipes
// (hg_exact.cuh), and what is monotone is taken once per trajectory: the root
// of the least squared distance, the quotient of the largest |C - C0|.
// The chunks' results meet in the outputs as integers: non-negative doubles
// order like their bit patterns, in which a NaN is above everything.
struct FilterSample {
  double q1, q2;  // squared distances to the primaries
  double C;       // Jacobi constant
};

__device__ __forceinline__ FilterSample filter_sample(const hg::FusedOps& o, const double* s, long long ld, double mu,
                                                      double mu1) {
  FilterSample r;
  const double x = s[0], y = s[ld], z = s[2 * ld], vx = s[3 * ld], vy = s[4 * ld], vz = s[5 * ld];
  const double a = o.add(x, mu), b = o.add(o.add(x, -o.one), mu), f = o.sub(x, mu1);
  const double yy = o.mul(y, y), zz = o.mul(z, z);
  auto square_sum = [&](double u) { return o.add(o.add(o.mul(u, u), yy), zz); };
  r.q1 = square_sum(a);
  r.q2 = square_sum(b);
  const double r1 = hg_sqrt(r.q1), r2 = hg_sqrt(square_sum(f));
  // (the doubled sum is exact: one rounding)
  r.C = o.sub(fma(o.add(hg_div(mu1, r1), hg_div(mu, r2)), 2.0, o.add(o.mul(x, x), yy)),
              o.add(o.add(o.mul(vx, vx), o.mul(vy, vy)), o.mul(vz, vz)));
  return r;
}

__device__ __forceinline__ unsigned long long pattern(double v) { return (unsigned long long)__double_as_longlong(v); }

// The reference's running minimum keeps a first NaN and passes over later
// ones; its running maximum starts at 0 and passes over NaN.
__device__ __forceinline__ void filter_finish(const FilterSample& first, unsigned long long q1, unsigned long long q2,
                                              unsigned long long e, double* min_r1, double* min_r2,
                                              double* max_rel_e) {
  const double absC0 = fabs(first.C), d = __longlong_as_double((long long)e);
  const double rel = absC0 > 1e-14 ? d / absC0 : d;
  *min_r1 = first.q1 != first.q1 ? first.q1 : sqrt(__longlong_as_double((long long)q1));
  *min_r2 = first.q2 != first.q2 ? first.q2 : sqrt(__longlong_as_double((long long)q2));
  *max_rel_e = rel > 0.0 ? rel : 0.0;
}

constexpr int kFilterBlock = 64;
constexpr int kFilterChunk = 16;  // least samples per chunk: each one also forms C of sample 0

// ONE: a single chunk, finished here; else the outputs hold bit patterns.
template <bool ONE>
__global__ void __launch_bounds__(kFilterBlock) filters_kernel(int N, int m, int chunk, const double* samples,
                                                               long long ld, double mu, double* min_r1,
                                                               double* min_r2, double* max_rel_e) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const double mu1 = 1.0 - mu;
  const hg::FusedOps o;
  const FilterSample first = filter_sample(o, samples + i, ld, mu, mu1);
  unsigned long long q1 = pattern(first.q1), q2 = pattern(first.q2), e = 0;
  const int lo = max(1, (int)blockIdx.y * chunk), hi = min(m, ((int)blockIdx.y + 1) * chunk);
  for (int q = lo; q < hi; ++q) {
    const FilterSample s = filter_sample(o, samples + (long long)q * 6 * ld + i, ld, mu, mu1);
    const unsigned long long p1 = pattern(s.q1), p2 = pattern(s.q2), d = pattern(fabs(o.sub(s.C, first.C)));
    q1 = p1 < q1 ? p1 : q1;
    q2 = p2 < q2 ? p2 : q2;
    e = d > e && d <= 0x7FF0000000000000ull ? d : e;
  }
  if constexpr (ONE) {
    filter_finish(first, q1, q2, e, min_r1 + i, min_r2 + i, max_rel_e + i);
  } else {
    atomicMin((unsigned long long*)min_r1 + i, q1);
    atomicMin((unsigned long long*)min_r2 + i, q2);
    atomicMax((unsigned long long*)max_rel_e + i, e);
  }
}

__global__ void filters_init_kernel(int N, double* min_r1, double* min_r2, double* max_rel_e) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  ((unsigned long long*)min_r1)[i] = ((unsigned long long*)min_r2)[i] = ~0ull;
  ((unsigned long long*)max_rel_e)[i] = 0ull;
}

__global__ void filters_finish_kernel(int N, const double* samples, long long ld, double mu, double* min_r1,
                                      double* min_r2, double* max_rel_e) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const FilterSample first = filter_sample(hg::FusedOps(), samples + i, ld, mu, 1.0 - mu);
  filter_finish(first, pattern(min_r1[i]), pattern(min_r2[i]), pattern(max_rel_e[i]), min_r1 + i, min_r2 + i,
                max_rel_e + i);
}

}  // namespace

extern "C" int hg_trajectory_filters(int N, int m, const double* samples, long long ld, double mu, double* min_r1,
                                     double* min_r2, double* max_rel_energy, void* stream) {
  if (N < 0 || m < 1 || ld < N) return HG_ERR_ARGS;
  if (N > 0 && (!samples || !min_r1 || !min_r2 || !max_rel_energy)) return HG_ERR_ARGS;
  if (N == 0) return HG_OK;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return HG_ERR_CUDA;
  const cudaStream_t st = (cudaStream_t)stream;
  // chunks: about 24 warps per SM in all
  const int bx = (N + kFilterBlock - 1) / kFilterBlock;
  const int most = (m + kFilterChunk - 1) / kFilterChunk;
  const long long want = (12LL * sms + bx - 1) / bx;
  const int parts = (int)(want < most ? want : most);
  const int chunk = (m + parts - 1) / parts;
  if (parts <= 1) {
    filters_kernel<true><<<bx, kFilterBlock, 0, st>>>(N, m, m, samples, ld, mu, min_r1, min_r2, max_rel_energy);
  } else {
    const int bi = (N + 127) / 128;
    filters_init_kernel<<<bi, 128, 0, st>>>(N, min_r1, min_r2, max_rel_energy);
    filters_kernel<false><<<dim3((unsigned)bx, (unsigned)((m + chunk - 1) / chunk)), kFilterBlock, 0, st>>>(
        N, m, chunk, samples, ld, mu, min_r1, min_r2, max_rel_energy);
    filters_finish_kernel<<<bi, 128, 0, st>>>(N, samples, ld, mu, min_r1, min_r2, max_rel_energy);
  }
  return cudaGetLastError() == cudaSuccess ? HG_OK : HG_ERR_CUDA;
}

extern "C" int hg_section_detect(int N, int m, const double* samples, long long ld, const double* times,
                                 long long times_ld, int axis, double offset, int direction, int plane_u,
                                 int plane_v, int segment_refine, int cubic, int newton_max_iter,
                                 double tol_on_surface, double dedup_time_tol, double dedup_point_tol, int max_hits,
                                 double* hit_t, double* hit_y, int* n_hits, int* n_found, void* stream) {
  if (N < 0 || m < 0 || ld < N || (times_ld != 0 && times_ld < N)) return HG_ERR_ARGS;
  if (axis < 0 || axis > 5 || plane_u < 0 || plane_u > 5 || plane_v < 0 || plane_v > 5) return HG_ERR_ARGS;
  if (direction < -1 || direction > 1 || segment_refine < 1 || max_hits < 1 || newton_max_iter < 0) return HG_ERR_ARGS;
  if (N > 0 && (!samples || !times || !hit_t || !hit_y || !n_hits)) return HG_ERR_ARGS;
  if (N == 0) return HG_OK;
  SecParams p;
  p.N = N;
  p.m = m;
  p.samples = samples;
  p.ld = ld;
  p.times = times;
  p.times_ld = times_ld;
  p.axis = axis;
  p.offset = offset;
  p.direction = direction;
  p.pu = plane_u;
  p.pv = plane_v;
  p.segment_refine = segment_refine;
  p.cubic = cubic ? 1 : 0;
  p.newton_max_iter = newton_max_iter;
  p.tol_on_surface = tol_on_surface;
  p.dedup_time_tol = dedup_time_tol;
  p.dedup_point_tol = dedup_point_tol;
  p.max_hits = max_hits;
  p.hit_t = hit_t;
  p.hit_y = hit_y;
  p.n_hits = n_hits;
  p.n_found = n_found;
  section_kernel<<<(N + kSecBlock - 1) / kSecBlock, kSecBlock, 0, (cudaStream_t)stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? HG_OK : HG_ERR_CUDA;
}
