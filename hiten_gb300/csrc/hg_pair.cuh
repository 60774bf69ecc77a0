// Layouts of the 42-dim variational system on several warps: fixed-step RK
// (fixed_rk_pair_kernel, fixed_rk_trio_kernel) and single-pass DOP853 without
// an event (dop853_pair_kernel, dop853_quad_kernel).
//
// Why.  On GB300 a warp has one FP64 instruction in flight at a time, for
// 64 cycles whatever the number of active lanes (76 when four warps share the
// SM's FP64 unit), so one warp's step costs (its FP64 instructions) x 64-76
// cycles.  A batch of about a thousand 42-dim trajectories gives only a few
// warps per SM, and its time is the per-warp instruction count of a step.
// The state of a trajectory (6 components, the Hessian of the potential and
// the accelerations) and its STM (36 components, F(x) Phi) are two
// instruction streams; run on two warps of one block they split that count.
//
// Layout.  A trajectory group is five trajectories served by two warps:
//   * the state warp: lane 6t + j (t < 5, j < 6) holds state component 36 + j
//     of trajectory t and does job j of the shared Hessian (hessian_job);
//     lanes 30 and 31 shadow group 4 (they repeat job 0 and write nothing);
//   * the STM warp: lane 6t + c holds column c of Phi (components 6r + c,
//     r = 0..5); lanes 30 and 31 shadow column 5 of trajectory 4.
// At every right-hand-side evaluation the state warp forms the Hessian's
// six entries from its stage state (the off-diagonal ones as the products
// hessian42 takes) and hands them to the STM warp through shared memory: a
// ring of kPairSlots slots with an mbarrier pair per slot, "full" after the state warp wrote
// it, "empty" after the STM warp read it; meanwhile the STM warp forms its
// stage columns.  Every operation and operand is the one the 7-lane layout
// uses (Layout<7>), so the results are bit-identical.
//
// Waits are bounded: a hand-off that has not completed within
// kPairWaitNs of wall time marks the warp broken; it stops waiting and
// arriving, the partner's waits run out in turn, both leave the step loop
// and the group's trajectories report HG_SYNC_TIMEOUT.
#pragma once

#include "hg_kernels.cuh"

namespace hg {

constexpr unsigned long long kPairWaitNs = 2000000000ull;  // 2 s per hand-off
constexpr int kPairTraj = 5;                                // trajectories per warp pair
constexpr unsigned kPairSlots = 4;                          // hand-off ring depth

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
  [[maybe_unused]] unsigned long long state;
  asm volatile("mbarrier.arrive.shared::cta.b64 %0, [%1];" : "=l"(state) : "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_test(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for the completion of the phase with the given parity; false when it
// has not completed within limit_ns (or 2^30 polls).
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity,
                                          unsigned long long limit_ns = kPairWaitNs) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  for (unsigned it = 1; it < (1u << 30); ++it) {
    if (mbar_test(bar, parity)) return true;
    if ((it & 63u) == 0 && global_ns() - t0 > limit_ns) return false;
  }
  return false;
}

// Self-test of the bounded wait (one block of two warps): warp 0 waits on a
// barrier that nothing arrives at and must give up after limit_ns; then warp
// 1 arrives at a second barrier and warp 0's wait on it must succeed.
// out[0] = 1 if the first wait ran out, out[1] = 1 if the second completed,
// out[2] = elapsed nanoseconds of the first wait.
static __global__ void bounded_wait_selftest_kernel(int* out, unsigned long long limit_ns) {
  __shared__ unsigned long long bars[2];
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 32);
    mbar_init(&bars[1], 32);
  }
  __syncthreads();
  const int w = threadIdx.x >> 5;
  if (w == 0) {
    const unsigned long long t0 = global_ns();
    const bool ok0 = mbar_wait(&bars[0], 0, limit_ns);  // nothing arrives
    const unsigned long long dt = global_ns() - t0;
    const bool ran_out = !__any_sync(0xFFFFFFFFu, ok0);
    const bool ok1 = __all_sync(0xFFFFFFFFu, mbar_wait(&bars[1], 0, limit_ns));
    if (threadIdx.x == 0) {
      out[0] = ran_out ? 1 : 0;
      out[1] = ok1 ? 1 : 0;
      out[2] = (int)(dt > 2000000000ull ? 2000000000ull : dt);
    }
  } else {
    mbar_arrive(&bars[1]);
  }
}

// Shared-memory hand-off of one warp pair.
struct PairLink {
  double H[kPairSlots][kPairTraj][8];  // slot, trajectory, (xx, yy, zz, xy, yz, xz, -, -)
  unsigned long long full[kPairSlots];
  unsigned long long empty[kPairSlots];
  int fin[kPairTraj];     // STM columns finite, per trajectory
  int broken;             // STM warp gave up a wait
};

// Lane placement shared by both warps of a pair.
struct PairLane {
  int t;           // trajectory in the group (0..4)
  int role;        // 0..5; 6 and 7 on the shadow lanes 30, 31
  int base;        // first lane of the trajectory
  unsigned gmask;  // lanes of the trajectory (group 4 includes the shadows)
  __device__ __forceinline__ explicit PairLane(int lane) {
    t = lane < 30 ? lane / 6 : 4;
    role = lane < 30 ? lane % 6 : lane - 24;
    base = 6 * t;
    gmask = t < 4 ? (0x3Fu << base) : 0xFF000000u;
  }
};

// State warp: one state component per lane (NC = 1).  Its stage sums are plain
// in the layouts whose chain it is, and three-register multiply-adds (OPS) beside
// one STM warp, where a filled SM's FP64 unit sets the time: 8192 trajectories,
// RK8 159 -> 150 us a step, DOP853 178 -> 176.
template <class OPS>
struct PairState {
  using Ops = OPS;
  Ops ops;
  static constexpr int D = 42;
  static constexpr int NC = 1;
  static constexpr bool kState = true;
  __device__ __forceinline__ int flag_slot() const { return 42; }  // gather-slot flag entry
  int role, base, t;
  unsigned gmask;
  PairLink* link;
  mutable unsigned seq;  // right-hand-side evaluations so far
  mutable bool broken;
  __device__ __forceinline__ int comp(int) const { return 36 + (role < 6 ? role : 0); }
  __device__ __forceinline__ double from(double v, int r) const { return __shfl_sync(gmask, v, base + r); }
  __device__ __forceinline__ void rhs(const double (&v)[1], double mu, const Dir& dir, double (&dv)[1]) const {
    const int job = role < 6 ? role : 0;  // (the shadow lanes repeat job 0 in full)
    const double x = from(v[0], 0), y = from(v[0], 1), z = from(v[0], 2);
    // position lanes: their derivative is the velocity of lane job + 3; lane 3
    // takes vy, lane 4 vx
    const double u = from(v[0], nibble(0x534543u, job));
    double off;
    const double form = hessian_job(job, x, y, z, u, mu, off);
    const unsigned b = seq % kPairSlots, use = seq / kPairSlots;
    if (!broken && use >= 1) {
      // the slot's previous contents must have been read (a warp-uniform outcome)
      const bool ok = mbar_wait(&link->empty[b], (use - 1u) & 1u);
      broken = !__all_sync(0xFFFFFFFFu, ok);
    }
    if (!broken) {
      // the six Hessian entries xx, yy, zz, xy, yz, xz
      if (role < 6) link->H[b][t][role] = role < 3 ? form : off;
      mbar_arrive(&link->full[b]);
    }
    ++seq;
    const double d = job < 3 ? u : form;
    const int c = comp(0);
    dv[0] = neg_if(d, c >= dir.neg_lo && c < dir.neg_hi);
  }
  static __device__ __forceinline__ int nibble(unsigned table, int job) { return (int)(table >> (4 * job)) & 7; }
  // hessian_split's work with each lane keeping its own entry: returns xx, yy,
  // zz, ax, ay, az for jobs 0..5 and sets `off` to xy, yz, xz on jobs 3..5.
  // Lane 3 b + k (b = primary, k < 3) takes the power of its primary its two
  // quotients divide by:
  //   0: mu2/r3, t1/r3     1: y/r3, z/r3     2: mu2/r5, (mu2 t1)/r5
  //   3: mu/R3,  t2/R3     4: y/R3, z/R3     5: mu/R5,  (mu t2)/R5
  // A job needs four of the twelve, two for a sum (s1 + s2) and two as factors
  // (f1, f2); four shuffles hand them out, each lane offering in each the one
  // its readers want.  The expressions and operands are hessian42's (x - m == x +
  // (-m), (-a) u == -(a u), -0 + v == v, a + b == b + a): same bits.  `u`: vy
  // on job 3, vx on job 4.  The state warp's chain is what a step of the trio
  // waits for (its STM warps alone would take 23.3 us of an RK8 step's 28.9):
  // twelve shuffles here and in rhs instead of the 26 of hessian_split and its
  // caller, and their selects, took it to 26.7 us.
  __device__ __forceinline__ double hessian_job(int job, double x, double y, double z, double u, double mu,
                                                double& off) const {
    const double mu2 = 1.0 - mu;
    const bool acc = job >= 3;
    const int k = acc ? job - 3 : job;
    const double m = acc ? mu : mu2;
    const double tt = x + (acc ? -mu2 : mu);  // x + mu | x - mu2
    // job 0: t1^2, 1: y^2, 2: mu2 t1, 3: t2^2, 4: z^2, 5: mu t2
    const double sq = (k == 0 ? tt : (job == 1 ? y : (job == 4 ? z : m))) * (job == 1 ? y : (job == 4 ? z : tt));
    const double ts = from(sq, acc ? 3 : 0);
    const double ys = from(sq, 1), zs = from(sq, 4);
    const double t2s = from(sq, 3);
    const double rr = (ts + ys) + zs;
    const double den = hg_power_of_r2(rr, k == 2);  // r^3, on jobs 2 and 5 r^5
    const double num[2] = {k == 1 ? y : m, k == 0 ? tt : (k == 1 ? z : sq)};
    double q[2];
    hg_quotients(num, den, q);
    //            jobs 0..2 read   job 3          job 4          job 5
    // s1         0: mu2/r3        2: mu2 t1/r5   5: mu/R5       2: mu2 t1/r5
    // s2         3: mu/R3         5: mu t2/R5    2: mu2/r5      5: mu t2/R5
    // f1         2: mu2/r5        0: t1/r3       1: y/r3        4: z/R3
    // f2         5: mu/R5         3: t2/R3       4: y/R3        1: z/r3
    const double s1 = from(job == 2 ? q[1] : q[0], nibble(0x252000u, job));
    const double s2 = from(job == 5 ? q[1] : q[0], nibble(0x525333u, job));
    const double f1 = from(job == 0 || job == 4 ? q[1] : q[0], nibble(0x410222u, job));
    const double f2 = from(job == 1 || job == 3 ? q[1] : q[0], nibble(0x143555u, job));
    // jobs 0..2: mu2/r5 3; the Coriolis term 2 vy, -2 vx on jobs 3, 4
    const double a = (acc ? (job == 4 ? -2.0 : 2.0) : f1) * (acc ? u : 3.0);
    // jobs 0..2: mu/R5 3; jobs 3..5: 3y, 3y, 3z of the off-diagonal entry
    const double b = (acc ? (job == 5 ? z : y) : f2) * 3.0;
    const double s = s1 + s2;
    double P, A, U, B, W, C;
    if (!acc) {
      P = job == 2 ? -0.0 : 1.0;
      A = a;
      U = job == 0 ? ts : (job == 1 ? ys : zs);
      B = b;
      W = job == 0 ? t2s : (job == 1 ? ys : zs);
      C = -s;
    } else {
      P = job == 3 ? x : (job == 4 ? y : -0.0);
      A = job == 5 ? -mu : -mu2;
      U = f1;
      B = job == 5 ? -mu2 : -mu;
      W = f2;
      C = job == 5 ? -0.0 : a;
    }
    const double form = ((P + A * U) + B * W) + C;
    // one product ((3a) b) c: (3y)(s) | ((3y) z)(s) | (3z)(s) (c = 1.0 exact)
    off = (b * (job == 4 ? z : s)) * (job == 4 ? s : 1.0);
    return form;
  }
};

// STM warp: one column of Phi per lane (NC = 6, rows 0..5).
struct PairStm {
  using Ops = FusedOps;
  Ops ops;
  static constexpr int D = 42;
  static constexpr int NC = 6;
  static constexpr bool kState = false;
  __device__ __forceinline__ int flag_slot() const { return 43; }  // and 44: the whole STM
  int col, t;
  int role, base;  // lane placement (role 0..7, as in the state warp), for group-wide steps
  unsigned gmask;
  PairLink* link;
  mutable unsigned seq;
  mutable bool broken;
  __device__ __forceinline__ int comp(int r) const { return 6 * r + col; }
  __device__ __forceinline__ void rhs(const double (&v)[6], double mu, const Dir& dir, double (&dv)[6]) const {
    (void)mu;
    const unsigned b = seq % kPairSlots;
    double xx = 0.0, yy = 0.0, zz = 0.0, xy = 0.0, xz = 0.0, yz = 0.0;
    if (!broken) {
      const bool ok = mbar_wait(&link->full[b], (seq / kPairSlots) & 1u);
      broken = !__all_sync(0xFFFFFFFFu, ok);
    }
    if (!broken) {
      const double* e = link->H[b][t];
      xx = e[0];
      yy = e[1];
      zz = e[2];
      xy = e[3];
      yz = e[4];
      xz = e[5];
      mbar_arrive(&link->empty[b]);
    }
    ++seq;
    // rows of F(x) @ Phi[:, col] (dynamics/rtbp.py:204-209), as Layout<7>
    dv[0] = v[3];
    dv[1] = v[4];
    dv[2] = v[5];
    // (the doubled velocities are exact: one rounding)
    const Ops& o = ops;
    dv[3] = fma(2.0, v[4], o.add(o.add(o.mul(xx, v[0]), o.mul(xy, v[1])), o.mul(xz, v[2])));
    dv[4] = fma(-2.0, v[3], o.add(o.add(o.mul(xy, v[0]), o.mul(yy, v[1])), o.mul(yz, v[2])));
    dv[5] = o.add(o.add(o.mul(xz, v[0]), o.mul(yz, v[1])), o.mul(zz, v[2]));
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      const int c = comp(r);
      dv[r] = neg_if(dv[r], c >= dir.neg_lo && c < dir.neg_hi);
    }
  }
};

// Half-column STM warps of the three-warp layout (fixed_rk_trio_kernel): two
// warps share the 36 STM components of five trajectories.  A half-group of
// six lanes holds three columns of one trajectory (columns 3 half .. 3 half +
// 2), each column on a lane pair as in Layout<14>: the even lane rows 0..2,
// the odd lane rows 3..5; warp w holds half-groups 5w .. 5w + 4 (trajectory
// = half-group / 2, half = half-group % 2).
struct PairStmHalf {
  using Ops = FusedOps;
  Ops ops;
  static constexpr int D = 42;
  static constexpr int NC = 3;
  static constexpr bool kState = false;
  int t, half;
  int role, base;  // lane placement within the half-group (6, 7 on the shadow lanes)
  unsigned gmask;
  PairLink* link;
  mutable unsigned seq;
  mutable bool broken;
  __device__ __forceinline__ int comp(int r) const {
    const int r6 = role % 6;
    return 6 * (3 * (r6 & 1) + r) + 3 * half + (r6 >> 1);
  }
  __device__ __forceinline__ void rhs(const double (&v)[3], double mu, const Dir& dir, double (&dv)[3]) const {
    (void)mu;
    const unsigned b = seq % kPairSlots;
    double xx = 0.0, yy = 0.0, zz = 0.0, xy = 0.0, xz = 0.0, yz = 0.0;
    if (!broken) {
      const bool ok = mbar_wait(&link->full[b], (seq / kPairSlots) & 1u);
      broken = !__all_sync(0xFFFFFFFFu, ok);
    }
    if (!broken) {
      const double* e = link->H[b][t];
      xx = e[0];
      yy = e[1];
      zz = e[2];
      xy = e[3];
      yz = e[4];
      xz = e[5];
      mbar_arrive(&link->empty[b]);
    }
    ++seq;
    // the partner lane (lane ^ 1) holds the other rows of the column
    const double q0 = __shfl_xor_sync(gmask, v[0], 1), q1 = __shfl_xor_sync(gmask, v[1], 1),
                 q2 = __shfl_xor_sync(gmask, v[2], 1);
    // rows 3..5 of F(x) Phi[:, c] (dynamics/rtbp.py:204-209), as Layout<14>:
    // the odd lane forms row 3, the even lane row 4 in the same instructions
    // and hands it over; both form row 5
    const bool pos = ((role % 6) & 1) == 0;
    const double p0 = pos ? v[0] : q0, p1 = pos ? v[1] : q1, p2 = pos ? v[2] : q2;
    const double w = pos ? q0 : v[1];  // row 3 takes 2 v4, row 4 -2 v3
    const Ops& o = ops;
    const double r34 = fma(pos ? -2.0 : 2.0, w, o.add(o.add(o.mul(pos ? xy : xx, p0), o.mul(pos ? yy : xy, p1)),
                                                      o.mul(pos ? yz : xz, p2)));
    const double r4 = __shfl_xor_sync(gmask, r34, 1);
    const double r5 = o.add(o.add(o.mul(xz, p0), o.mul(yz, p1)), o.mul(zz, p2));
    const double d0 = pos ? q0 : r34, d1 = pos ? q1 : r4, d2 = pos ? q2 : r5;
    dv[0] = neg_if(d0, comp(0) >= dir.neg_lo && comp(0) < dir.neg_hi);
    dv[1] = neg_if(d1, comp(1) >= dir.neg_lo && comp(1) < dir.neg_hi);
    dv[2] = neg_if(d2, comp(2) >= dir.neg_lo && comp(2) < dir.neg_hi);
  }
};

// Third-column STM warps of the four-warp layout: three warps share the 36 STM
// components of five trajectories.  A third-group of six lanes holds two
// columns of one trajectory, each on three lanes: lane i of a column holds its
// rows i and 3 + i.  The derivative of row i is the lane's own row 3 + i, and
// lane i forms row 3 + i of F(x) Phi[:, c] from rows 0..2 (its own and the two
// other lanes') and its row of the Hessian: six FP64 instructions a
// right-hand side where the half column's lanes take eleven.  Warp w holds
// third-groups 5w .. 5w + 4 (trajectory = third-group / 3).  A third-group is a
// complete six-lane group for the step control (coefficients, norms, step-size
// factor), so a trajectory's three parts take the same decisions.
struct PairStmThird {
  using Ops = FusedOps;
  Ops ops;
  static constexpr int D = 42;
  static constexpr int NC = 2;
  static constexpr bool kState = false;
  int t, part;     // part 0..2: columns 2 part, 2 part + 1
  int role, base;  // lane placement within the third-group (6, 7 on the shadow lanes)
  unsigned gmask;
  PairLink* link;
  mutable unsigned seq;
  mutable bool broken;
  __device__ __forceinline__ int flag_slot() const { return 43 + part; }
  __device__ __forceinline__ int row() const { return role % 3; }
  __device__ __forceinline__ int comp(int r) const { return 6 * (3 * r + role % 3) + 2 * part + (role % 6) / 3; }
  __device__ __forceinline__ double from(double v, int r) const { return __shfl_sync(gmask, v, r); }
  __device__ __forceinline__ void rhs(const double (&v)[2], double mu, const Dir& dir, double (&dv)[2]) const {
    (void)mu;
    const unsigned b = seq % kPairSlots;
    const int i = row();
    const int col = base + (role % 6) / 3 * 3;  // first lane of the column
    // rows 0..2 of the column, the paired velocity (row 3 takes 2 v4, row 4 -2 v3)
    const double p0 = from(v[0], col), p1 = from(v[0], col + 1), p2 = from(v[0], col + 2);
    const double w = from(v[1], col + (i == 0 ? 1 : 0));
    // this lane's row of the Hessian (xx, yy, zz, xy, yz, xz)
    double h0 = 0.0, h1 = 0.0, h2 = 0.0;
    if (!broken) {
      const bool ok = mbar_wait(&link->full[b], (seq / kPairSlots) & 1u);
      broken = !__all_sync(0xFFFFFFFFu, ok);
    }
    if (!broken) {
      const double* e = link->H[b][t];
      h0 = e[i == 0 ? 0 : (i == 1 ? 3 : 5)];
      h1 = e[i == 0 ? 3 : (i == 1 ? 1 : 4)];
      h2 = e[i == 0 ? 5 : (i == 1 ? 4 : 2)];
      mbar_arrive(&link->empty[b]);
    }
    ++seq;
    const Ops& o = ops;
    const double s = o.add(o.add(o.mul(h0, p0), o.mul(h1, p1)), o.mul(h2, p2));
    // (the doubled velocities are exact: one rounding)
    const double c = fma(i == 0 ? 2.0 : -2.0, w, s);
    const double d1 = i == 2 ? s : c;
    dv[0] = neg_if(v[1], comp(0) >= dir.neg_lo && comp(0) < dir.neg_hi);
    dv[1] = neg_if(d1, comp(1) >= dir.neg_lo && comp(1) < dir.neg_hi);
  }
};

// One warp's part of a fixed-step propagation (rk.py:531-588): loads its
// components, steps through the nodes, writes rows 0, out_every, ...
// Returns whether its components stayed finite.
// `sm`: this warp's pair_fixed_doubles<ORDER>(NC) of shared memory (stage
// derivatives, the step's products).
template <int ORDER>
__host__ __device__ constexpr int pair_fixed_doubles(int nc) {
  return stage_slots<FixedTab<ORDER>>() * nc * 32 + stage_nnz<FixedTab<ORDER>>();
}
template <int ORDER, class LT>
__device__ __forceinline__ bool pair_fixed_run(const LT& L, const FixedParams& p, int traj, bool writes, double* sm) {
  constexpr int NC = LT::NC;
  double y[NC];
#pragma unroll
  for (int r = 0; r < NC; ++r) y[r] = p.y0[(long long)L.comp(r) * p.ld_in + traj];
  if (writes) {
#pragma unroll
    for (int r = 0; r < NC; ++r) p.out[(long long)L.comp(r) * p.ld_out + traj] = y[r];
  }
  const long long row = 42LL * p.ld_out;
  bool finite = true;
  using T = FixedTab<ORDER>;
  const StageMem<T, NC> k{sm + (threadIdx.x & 31)};
  TableCoef<T, 32, 1> cf{sm + StageMem<T, NC>::doubles, (int)(threadIdx.x & 31), 0xFFFFFFFFu};
  for (int idx = 0; idx < p.n - 1; ++idx) {
    const double h = p.t_vals[idx + 1] - p.t_vals[idx];
    cf.set_step(h);
    double yn[NC];
    rk_fixed_step_loop<ORDER>(L, y, cf, p.mu, p.dir, k, yn);
#pragma unroll
    for (int r = 0; r < NC; ++r) {
      y[r] = yn[r];
      finite = finite && finite_bits(yn[r]);
    }
    if (writes && (idx + 1) % p.out_every == 0) {
      double* o = p.out + (long long)((idx + 1) / p.out_every) * row;
#pragma unroll
      for (int r = 0; r < NC; ++r) o[(long long)L.comp(r) * p.ld_out + traj] = y[r];
    }
    if (L.broken) break;
  }
  return finite;
}

template <int ORDER>
__host__ __device__ constexpr size_t pair_fixed_smem(int block) {
  return (size_t)(block / 64) * (pair_fixed_doubles<ORDER>(1) + pair_fixed_doubles<ORDER>(6)) * sizeof(double);
}

// Blocks of 2P warps (P = blockDim.x / 64 pairs): warps 0..P-1 are the state
// warps of pairs 0..P-1, warps P..2P-1 their STM warps, so each warp of a
// four-warp block lands on its own sub-partition.
template <int ORDER>
__global__ void __launch_bounds__(128) fixed_rk_pair_kernel(FixedParams p) {
  __shared__ PairLink links[2];
  extern __shared__ double sm_step[];  // pair_fixed_smem<ORDER>(blockDim.x)
  const int w = threadIdx.x >> 5;
  const int npairs = blockDim.x >> 6;
  const int pair = w % npairs;
  const bool stm = w >= npairs;
  const int lane = threadIdx.x & 31;
  PairLink* lk = &links[pair];
  if (threadIdx.x < npairs * (int)kPairSlots) {
    PairLink* l = &links[threadIdx.x / kPairSlots];
    const int s = threadIdx.x % kPairSlots;
    mbar_init(&l->full[s], 32);
    mbar_init(&l->empty[s], 32);
    if (s == 0) l->broken = 0;
  }
  __syncthreads();
  const PairLane pl(lane);
  const int group = blockIdx.x * npairs + pair;
  const bool active = group * kPairTraj < p.N;  // uniform over the pair's two warps
  const int traj = group * kPairTraj + pl.t;
  const bool valid = active && traj < p.N;
  const int tc = valid ? traj : (active ? p.N - 1 : 0);
  bool finite = true, broken = false;
  if (active) {
    if (!stm) {
      PairState<FusedOps> L;
      L.role = pl.role;
      L.base = pl.base;
      L.t = pl.t;
      L.gmask = pl.gmask;
      L.link = lk;
      L.seq = 0;
      L.broken = false;
      finite = pair_fixed_run<ORDER>(L, p, tc, valid && pl.role < 6, sm_step + pair * pair_fixed_doubles<ORDER>(1));
      broken = L.broken;
      finite = __all_sync(pl.gmask, finite);
    } else {
      PairStm L;
      L.col = pl.role < 6 ? pl.role : 5;
      L.t = pl.t;
      L.role = pl.role;
      L.base = pl.base;
      L.gmask = pl.gmask;
      L.link = lk;
      L.seq = 0;
      L.broken = false;
      finite = pair_fixed_run<ORDER>(L, p, tc, valid && pl.role < 6,
                                     sm_step + npairs * pair_fixed_doubles<ORDER>(1) + pair * pair_fixed_doubles<ORDER>(6));
      broken = L.broken;
      finite = __all_sync(pl.gmask, finite);
      if (pl.role == 0) lk->fin[pl.t] = finite ? 1 : 0;
      if (broken && lane == 0) lk->broken = 1;
    }
  }
  __syncthreads();
  if (!stm && valid && pl.role == 0 && p.status) {
    const bool all_fin = finite && lk->fin[pl.t] != 0;
    p.status[traj] = (broken || lk->broken) ? HG_SYNC_TIMEOUT : (all_fin ? HG_OK : HG_NONFINITE);
  }
}

// Three-warp fixed-step RK (42-dim, no event): blocks of 96 threads, warp 0
// the state warp of five trajectories, warps 1 and 2 their STM as half
// columns (PairStmHalf).  The STM warp's stage work is halved and a batch of N
// trajectories issues 3N / 5 warps instead of 2N / 5: an RK8 step 26.8 us
// against the pair's 41.4 while every SM holds one group, 30.6 / 41.7 with two,
// 41.2 / 42.9 with three, behind beyond (the groups share an SM's FP64 unit).
// The Hessian ring's "empty" barriers take both STM warps' arrivals.
template <int ORDER>
__host__ __device__ constexpr size_t trio_fixed_smem() {
  return (size_t)(pair_fixed_doubles<ORDER>(1) + 2 * pair_fixed_doubles<ORDER>(3)) * sizeof(double);
}
template <int ORDER>
__global__ void __launch_bounds__(96) fixed_rk_trio_kernel(FixedParams p) {
  __shared__ PairLink link;
  extern __shared__ double sm_step[];  // trio_fixed_smem<ORDER>()
  __shared__ int fin_half[kPairTraj][2];
  const int w = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < (int)kPairSlots) {
    mbar_init(&link.full[threadIdx.x], 32);
    mbar_init(&link.empty[threadIdx.x], 64);
    if (threadIdx.x == 0) link.broken = 0;
  }
  if (threadIdx.x < 2 * kPairTraj) fin_half[threadIdx.x >> 1][threadIdx.x & 1] = 1;
  __syncthreads();
  const PairLane pl(lane);
  const int group = blockIdx.x;
  const bool active = group * kPairTraj < p.N;  // uniform over the block
  const int hg = 5 * (w - 1) + pl.t;            // STM warps: half-group 0..9
  const int tg = w == 0 ? pl.t : hg / 2;
  const int traj = group * kPairTraj + tg;
  const bool valid = active && traj < p.N;
  const int tc = valid ? traj : (active ? p.N - 1 : 0);
  bool finite = true, broken = false;
  if (active) {
    if (w == 0) {
      PairState<PlainOps> L;
      L.role = pl.role;
      L.base = pl.base;
      L.t = pl.t;
      L.gmask = pl.gmask;
      L.link = &link;
      L.seq = 0;
      L.broken = false;
      finite = pair_fixed_run<ORDER>(L, p, tc, valid && pl.role < 6, sm_step);
      broken = L.broken;
      finite = __all_sync(pl.gmask, finite);
    } else {
      PairStmHalf L;
      L.t = tg;
      L.half = hg & 1;
      L.role = pl.role;
      L.base = pl.base;
      L.gmask = pl.gmask;
      L.link = &link;
      L.seq = 0;
      L.broken = false;
      finite = pair_fixed_run<ORDER>(L, p, tc, valid && pl.role < 6,
                                     sm_step + pair_fixed_doubles<ORDER>(1) + (w - 1) * pair_fixed_doubles<ORDER>(3));
      broken = L.broken;
      finite = __all_sync(pl.gmask, finite);
      if (pl.role == 0) fin_half[tg][hg & 1] = finite ? 1 : 0;
      if (broken && lane == 0) link.broken = 1;
    }
  }
  __syncthreads();
  if (w == 0 && valid && pl.role == 0 && p.status) {
    const bool all_fin = finite && fin_half[pl.t][0] != 0 && fin_half[pl.t][1] != 0;
    p.status[traj] = (broken || link.broken) ? HG_SYNC_TIMEOUT : (all_fin ? HG_OK : HG_NONFINITE);
  }
}

// ---------------------------------------------------------------------------
// DOP853 on the paired warps (42-dim, single pass, no event; rk.py:2375-2549)
// ---------------------------------------------------------------------------
// Besides the Hessian hand-off, the step-size control needs norms over all
// 42 components: both warps store their components of two vectors (and one
// flag each) in a per-trajectory gather slot, meet at a two-warp barrier (an
// mbarrier with 64 arrivals, two slots alternating by exchange), and every
// lane then forms the same numpy-order dots -- so both warps take the same
// accept / reject decisions, step sizes and dense-output samples.  Each warp
// loops while any of its five trajectories is running; finished ones keep
// computing on their frozen state without committing anything, so every
// hand-off has all 32 lanes of both warps.
struct PairGather {
  // slot, trajectory, vector, 42 components + flags: [42] the state warp's,
  // [43..45] the STM's (one warp: all; three third-column warps: one each)
  double v[2][kPairTraj][2][46];
  unsigned long long bar[2];
};

template <class LT>
__device__ __forceinline__ void pair_exchange(const LT& L, PairGather* gx, unsigned& gseq,
                                              const double (&a)[LT::NC], const double (&b)[LT::NC],
                                              double flag, double& dot_a, double& dot_b, double& flag_all) {
  const unsigned sl = gseq & 1u;
  double* va = gx->v[sl][L.t][0];
  double* vb = gx->v[sl][L.t][1];
  if (!L.broken) {
    if (L.role < 6) {
#pragma unroll
      for (int r = 0; r < LT::NC; ++r) {
        va[L.comp(r)] = a[r];
        vb[L.comp(r)] = b[r];
      }
      if (L.role == 0) {
        va[L.flag_slot()] = flag;
        if constexpr (!LT::kState && LT::NC == 6) va[44] = va[45] = flag;
      }
    }
    mbar_arrive(&gx->bar[sl]);
    const bool ok = mbar_wait(&gx->bar[sl], (gseq >> 1) & 1u);
    L.broken = !__all_sync(0xFFFFFFFFu, ok);
  }
  ++gseq;
  dots42_group(L, va, vb, dot_a, dot_b);
  flag_all = (va[42] != 0.0 && va[43] != 0.0 && va[44] != 0.0 && va[45] != 0.0) ? 1.0 : 0.0;
}

// Shared memory of a warp: stage derivatives, then its groups' products.
__host__ __device__ constexpr int pair_dop_doubles(int nc) {
  return stage_slots<DopTab>() * nc * 32 + stage_nnz<DopTab>() * kPairTraj;
}
// A pair's link, gather slots and both warps' parts.
__host__ __device__ constexpr size_t pair_dop_bytes() {
  return sizeof(PairLink) + sizeof(PairGather) + (pair_dop_doubles(1) + pair_dop_doubles(6)) * sizeof(double);
}
__host__ __device__ constexpr size_t pair_dop_smem(int block) { return (size_t)(block / 64) * pair_dop_bytes(); }
__host__ __device__ constexpr size_t quad_dop_smem() {
  return (size_t)(pair_dop_doubles(1) + 3 * pair_dop_doubles(2)) * sizeof(double);
}

// One warp's part of the DOP853 propagation of its five trajectories.
// Decisions that set how many hand-offs a step makes (keep stepping, build a
// dense cache) are votes over the warp (BLOCK = false: both warps of a pair
// hold the same trajectories) or over the block (BLOCK = true: the four
// warps of a quad hold different subsets).  Returns its broken flag.
template <bool BLOCK, class LT>
__device__ __forceinline__ bool pair_dop_run(const LT& L, const DopParams& p, PairGather* gx, double* sm, int traj,
                                             bool valid, bool writes) {
  auto vote_any = [](bool v) -> bool {
    if constexpr (BLOCK)
      return __syncthreads_or(v ? 1 : 0) != 0;
    else
      return __any_sync(0xFFFFFFFFu, v);
  };
  constexpr int NC = LT::NC;
  constexpr int D = 42;
  const double t0 = p.t0_arr ? p.t0_arr[traj] : p.t0;
  const double tmax = p.tmax_arr ? p.tmax_arr[traj] : p.tmax;
  double y[NC];
#pragma unroll
  for (int r = 0; r < NC; ++r) y[r] = p.y0[(long long)L.comp(r) * p.ld + traj];
  const StageMem<DopTab, NC> k{sm + (threadIdx.x & 31)};
  double k0[NC];
  L.rhs(y, p.mu, p.dir, k0);
#pragma unroll
  for (int d = 0; d < NC; ++d) k[0][d] = k0[d];
  unsigned gseq = 0;
  double h;
  {
    double a[NC], b[NC];
#pragma unroll
    for (int d = 0; d < NC; ++d) {
      const double scale0 = p.atol + p.rtol * fabs(y[d]);
      a[d] = y[d] / scale0;
      b[d] = k0[d] / scale0;
    }
    double da, db, unused;
    pair_exchange(L, gx, gseq, a, b, 0.0, da, db, unused);
    const double sn = sqrt((double)D);
    h = select_initial_step(sqrt(da) / sn, sqrt(db) / sn, p.min_step, p.max_step);
  }
  double t = t0, err_prev = -1.0, prev_pow = 0.0;
  int acc = 0, rej = 0;
  const bool dense = p.m >= 2;
  int q_next = (dense && p.dense_last) ? p.m - 1 : 0;
  int status = HG_OK;
  bool running = valid;
  double step_ls = 0.0;
  if (dense) step_ls = (tmax - t0) / (double)(p.m - 1);
  auto sample_t = [&](int q) -> double { return q == p.m - 1 ? tmax : (double)q * step_ls + t0; };
  // integrators/rk.py loop test (t - t_end) * direction < 0, direction +1
  bool live = running && hg_lt0(t - tmax);
  // (the shadow lanes of group 4 write their role's entries again)
  TableCoef<DopTab, 6, kPairTraj> cf{sm + StageMem<DopTab, NC>::doubles + L.base / 6, L.role % 6, L.gmask};
  while (vote_any(live)) {
    bool go = live;
    if (go && (long long)(acc + rej) >= p.max_steps) {
      status = HG_MAX_STEPS;
      running = false;
      go = false;
    }
    double hh = h;
    if (go) {
      hh = clamp_step(hh, p.max_step, p.min_step);
      hh = adjust_step_to_endpoint(t, hh, tmax);
    }
    double yh[NC], e5[NC], e3[NC];
    cf.set_step(hh);
    DopLaneT<LT>::step_loop(L, y, cf, hh, p.mu, p.dir, k, yh, e5, e3);
    double s5[NC], s3[NC];
    bool fin = true;
#pragma unroll
    for (int d = 0; d < NC; ++d) {
      const double scale = p.atol + p.rtol * np_maximum_abs(y[d], yh[d]);
      const double n53[2] = {e5[d], e3[d]};
      double q53[2];
      hg_quotients(n53, scale, q53);
      s5[d] = q53[0];
      s3[d] = q53[1];
      fin = fin && finite_bits(yh[d]);
    }
    fin = __all_sync(L.gmask, fin);
    double n5, n3, fin_all;
    pair_exchange(L, gx, gseq, s5, s3, fin ? 1.0 : 0.0, n5, n3, fin_all);
    fin = fin_all != 0.0;
    double err_norm;
    if (hg_both0(n5, n3))
      err_norm = 0.0;
    else
      err_norm = hg_div(fabs(hh) * n5, hg_sqrt((n5 + 0.01 * n3) * (double)D));
    const bool accepted = hg_le_pos(err_norm, HG_BITS_1);  // err_norm <= 1
    const double t_new = t + hh;
    // dense samples inside (t, t_new] (reference: searchsorted on nodes);
    // the cache's three extra evaluations run on the whole warp
    bool need = false, last = false;
    if (go && accepted && dense) {
      last = !(t_new - tmax < 0.0);
      need = q_next < p.m && (last || sample_t(q_next) < t_new);
    }
    if (vote_any(need)) {
      const double hseg = t_new - t;
      double F[7][NC];
      DopLaneT<LT>::dense_cache(L, y, yh, hseg, p.mu, p.dir, k, F);
      if (need) {
        while (q_next < p.m && (last || sample_t(q_next) < t_new)) {
          const double x = (sample_t(q_next) - t) / hseg;
          if (writes) {
            double* o = p.y_out + (long long)(p.dense_last ? 0 : q_next) * D * p.ld;
#pragma unroll
            for (int d = 0; d < NC; ++d) o[(long long)L.comp(d) * p.ld + traj] = DopLaneT<LT>::eval1(y[d], F, d, x);
          }
          ++q_next;
        }
      }
    }
    if (go) {
      if (accepted) {
        ++acc;
        t = t_new;
#pragma unroll
        for (int d = 0; d < NC; ++d) {
          y[d] = yh[d];
          k[0][d] = k[12][d];
        }
      } else {
        ++rej;
      }
      h = hh * pi_factor(L, accepted, err_norm, err_prev, prev_pow);
      if (accepted) {
        err_prev = err_norm;
        if (!fin) {
          status = HG_NONFINITE;
          running = false;
        }
      } else {
        h = clamp_step(h, p.max_step, p.min_step);
      }
    }
    live = running && hg_lt0(t - tmax) && !L.broken;
  }
  if (valid && writes) {
    // the reference's dense output falls back to the single stored node when
    // no step was taken
    if (dense) {
      while (q_next < p.m) {
        double* o = p.y_out + (long long)(p.dense_last ? 0 : q_next) * D * p.ld;
#pragma unroll
        for (int d = 0; d < NC; ++d) o[(long long)L.comp(d) * p.ld + traj] = y[d];
        ++q_next;
      }
    }
    if (p.y_end) {
#pragma unroll
      for (int d = 0; d < NC; ++d) p.y_end[(long long)L.comp(d) * p.ld + traj] = y[d];
    }
    if (LT::kState && L.role == 0) {
      if (p.t_end) p.t_end[traj] = t;
      if (p.n_accept) p.n_accept[traj] = acc;
      if (p.n_reject) p.n_reject[traj] = rej;
      if (p.status) p.status[traj] = status;
    }
  }
  return L.broken;
}

// Blocks of one or two pairs, laid out as fixed_rk_pair_kernel's.
// Six blocks of one pair per SM: 168 registers a thread (the dense cache of an
// STM column, built once or never per trajectory, spills 100 bytes) and 29.5 KB
// of shared memory; at the 255 registers taken unasked four blocks fit, and
// 4096 trajectories (5.4 groups per SM) took two rounds.
static __global__ void __launch_bounds__(128, 3) dop853_pair_kernel(DopParams p) {
  static_assert(sizeof(PairLink) % 8 == 0 && sizeof(PairGather) % 8 == 0, "");
  extern __shared__ double sm_step[];  // pair_dop_smem(blockDim.x): links, gathers, the warps' parts
  const int w = threadIdx.x >> 5;
  const int npairs = blockDim.x >> 6;
  const int pair = w % npairs;
  const bool stm = w >= npairs;
  const int lane = threadIdx.x & 31;
  PairLink* const links = (PairLink*)sm_step;
  PairGather* const gathers = (PairGather*)(links + npairs);
  double* const sm = (double*)(gathers + npairs);
  PairLink* lk = &links[pair];
  PairGather* gx = &gathers[pair];
  if (threadIdx.x < npairs * (int)kPairSlots) {
    PairLink* l = &links[threadIdx.x / kPairSlots];
    const int s = threadIdx.x % kPairSlots;
    mbar_init(&l->full[s], 32);
    mbar_init(&l->empty[s], 32);
    if (s == 0) l->broken = 0;
    if (s < 2) mbar_init(&gathers[threadIdx.x / kPairSlots].bar[s], 64);
  }
  __syncthreads();
  const PairLane pl(lane);
  const int group = blockIdx.x * npairs + pair;
  // list mode (n_in given): the trajectories 0 .. *n_in - 1 of a launch sized
  // for p.N run; the others' blocks return at once
  const int N = p.n_in ? *p.n_in : p.N;
  const bool active = group * kPairTraj < N;  // uniform over the pair's two warps
  const int traj = group * kPairTraj + pl.t;
  const bool valid = active && traj < N;
  const int tc = valid ? traj : (active ? N - 1 : 0);
  bool broken = false;
  if (active) {
    if (!stm) {
      PairState<FusedOps> L;
      L.role = pl.role;
      L.base = pl.base;
      L.t = pl.t;
      L.gmask = pl.gmask;
      L.link = lk;
      L.seq = 0;
      L.broken = false;
      broken = pair_dop_run<false>(L, p, gx, sm + pair * pair_dop_doubles(1), tc, valid, valid && pl.role < 6);
    } else {
      PairStm L;
      L.col = pl.role < 6 ? pl.role : 5;
      L.t = pl.t;
      L.role = pl.role;
      L.base = pl.base;
      L.gmask = pl.gmask;
      L.link = lk;
      L.seq = 0;
      L.broken = false;
      broken = pair_dop_run<false>(L, p, gx, sm + npairs * pair_dop_doubles(1) + pair * pair_dop_doubles(6), tc,
                                   valid, valid && pl.role < 6);
      if (broken && lane == 0) lk->broken = 1;
    }
  }
  __syncthreads();
  if (!stm && valid && pl.role == 0 && p.status && (broken || lk->broken)) p.status[traj] = HG_SYNC_TIMEOUT;
}

// Four-warp DOP853 (42-dim, single pass, no event): blocks of 128 threads,
// warp 0 the state warp of five trajectories, warps 1 to 3 their STM as thirds
// of columns (PairStmThird): two components a lane in the stage sums, the
// error norms and the quotients, where half columns on two warps hold three.
// A step of up to 760 trajectories took 36.4 us on three warps and takes 33.8;
// 1000 to 2048 trajectories (two or three groups an SM) are level, 40.4 and
// 53.  (Fixed steps, with neither norms nor quotients, keep half columns: 26.8 us
// a step on three warps, 28.1 on four, whose fourth warp only takes turns at
// the FP64 unit.)  The Hessian ring's "empty" barriers take the three STM warps'
// arrivals, the norm gather all four warps'.
static __global__ void __launch_bounds__(128) dop853_quad_kernel(DopParams p) {
  __shared__ PairLink link;
  __shared__ PairGather gather;
  extern __shared__ double sm_step[];  // quad_dop_smem()
  const int w = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < (int)kPairSlots) {
    mbar_init(&link.full[threadIdx.x], 32);
    mbar_init(&link.empty[threadIdx.x], 96);
    if (threadIdx.x < 2) mbar_init(&gather.bar[threadIdx.x], 128);
    if (threadIdx.x == 0) link.broken = 0;
  }
  __syncthreads();
  const PairLane pl(lane);
  const int group = blockIdx.x;
  // list mode (n_in given): the trajectories 0 .. *n_in - 1 run
  const int N = p.n_in ? *p.n_in : p.N;
  const bool active = group * kPairTraj < N;  // uniform over the block
  // trajectory of this lane within the group
  const int tp = 5 * (w - 1) + pl.t;  // STM warps: third-group 0..14
  const int tg = w == 0 ? pl.t : tp / 3;
  const int traj = group * kPairTraj + tg;
  const bool valid = active && traj < N;
  const int tc = valid ? traj : (active ? N - 1 : 0);
  bool broken = false;
  if (active) {
    if (w == 0) {
      PairState<PlainOps> L;
      L.role = pl.role;
      L.base = pl.base;
      L.t = pl.t;
      L.gmask = pl.gmask;
      L.link = &link;
      L.seq = 0;
      L.broken = false;
      broken = pair_dop_run<true>(L, p, &gather, sm_step, tc, valid, valid && pl.role < 6);
    } else {
      PairStmThird L;
      L.t = tg;
      L.part = tp % 3;
      L.role = pl.role;
      L.base = pl.base;
      L.gmask = pl.gmask;
      L.link = &link;
      L.seq = 0;
      L.broken = false;
      broken = pair_dop_run<true>(L, p, &gather, sm_step + pair_dop_doubles(1) + (w - 1) * pair_dop_doubles(2), tc, valid,
                                  valid && pl.role < 6);
      if (broken && lane == 0) link.broken = 1;
    }
  }
  __syncthreads();
  if (w == 0 && valid && pl.role == 0 && p.status && (broken || link.broken)) p.status[traj] = HG_SYNC_TIMEOUT;
}

}  // namespace hg
