// Section-point matching for heteroclinic connections
// (connections/backends.py:31-235): radius pairs between two 2-D point sets
// with each query point's nearest partner, and each set's nearest neighbour.
//
// Small sets are searched all-pairs, larger ones through a grid (below).  GB300
// retires FP32 ~60x faster than FP64, so every pair met is first screened in FP32
// with a margin that provably covers the FP32 rounding, and only the survivors
// are decided in FP64 with the
// reference's exact comparisons (dx*dx + dy*dy <= r^2, strict < for minima,
// the lower index winning ties).  Results are therefore those of the FP64
// loops.  Error bounds (u = 2^-24, R = max |coordinate| of both sets,
// a_f = fl32(a)): |a_f - a| <= u R; dx_f = fl32(a_f - b_f) satisfies
// |dx_f - dx| <= u|dx_f|(1 + 2u) + 2uR =: eta; d2_f = fl32(fl32(dx_f^2) +
// fl32(dy_f^2)) satisfies |d2_f - d2| <= 2^-21.8 d2_f + 2^-21.9 R(|dx_f| +
// |dy_f|) + 2^-45 R^2, bounded here by
//   e = 2^-20 (d2_f + R(|dx_f| + |dy_f|)) + 2^-43 R^2   (evaluated in FP32,
// the factor-two slack absorbing its own rounding).  Radius screen: a pair
// needs |dx|, |dy| <= eps, hence |dx_f|, |dy_f| <= T = (eps + 2^-22 R)(1 + 2^-20).
//
// Sets of more pairs (kNearestPairs, kRadiusPairs) are searched through a uniform
// grid over the reference points' bounding box, built in the same workspace: a
// query meets the points of the cells around it only, and a block scans all
// points for the few queries whose nearest one is many cells away.  Which pairs
// are decided, and how, stays as above, and the (d2, index) minimum and the count
// do not depend on the order, so the results do not either.  Points crowded into
// few cells (or coordinates that are not finite) leave the grid unused, by a
// count on the device.  65536 x 65536 points on two noisy curves, all pairs ->
// grid: radius 1.47 -> 0.18 ms, nearest 2.74 -> 0.18 ms, 0.06 of each the building.
#include <cuda_runtime.h>
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "hg_strided.cuh"
#include "hitengpu.h"

namespace {

constexpr int kTile = 256;
constexpr int kBlock = 128;

// One tile of reference points in shared memory: their FP32 copies for the
// screen (converted once per call by to_float2_kernel: a double-to-float
// conversion holds GB300's FP64 pipe, so converting in every block's tile load
// costs as much as the screen).  The exact FP64 decisions read the rare
// surviving points from global memory.
struct Tile {
  float2 f[kTile];
};

__device__ __forceinline__ void load_tile(Tile& T, const float2* __restrict__ pf, int base, int n) {
  for (int t = threadIdx.x; t < n; t += blockDim.x) T.f[t] = pf[base + t];
}

// The grid's numbers, in the last 256 bytes of the workspace's 8 n.  Where the
// grid is not used the FP32 copy takes their place too (the all-pairs scans have
// no registers to spare for points that it leaves out), so `use` is set by a
// pattern no FP32 copy has: two signalling NaNs, which no conversion returns.
constexpr int kHeadPoints = 32;
constexpr unsigned long long kUse = 0x7FA5A5A57FA5A5A5ull;
struct GridHead {
  unsigned long long lo[2], hi[2];  // bounding box as ordered keys
  unsigned long long work;          // candidates of all queries
  double x0, y0, inv, cell;         // cell of x: floor((x - x0) inv)
  unsigned long long use;           // kUse: search through the grid
  int far;                          // it left queries to nearest_far_kernel
  __device__ __forceinline__ bool used() const { return use == kUse; }
};
static_assert(sizeof(GridHead) <= 8 * kHeadPoints, "");

__global__ void to_float2_kernel(int n, const double* __restrict__ x, const double* __restrict__ y,
                                 float2* __restrict__ out, const GridHead* __restrict__ grid) {
  if (grid && grid->used()) {
    if (!grid->far) return;
    n -= kHeadPoints;
  }
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = make_float2((float)x[i], (float)y[i]);
}

// (d2, j) lexicographic minimum of two candidates (j < 0: none).  A scan in
// increasing j that keeps the first strict minimum ends at the lowest index
// of the minimal distance, which is this minimum over any split of the scan.
__device__ __forceinline__ void take_best(double& bd, int& bj, double d2, int j) {
  if (j >= 0 && (bj < 0 || d2 < bd || (d2 == bd && j < bj))) {
    bd = d2;
    bj = j;
  }
}

// The S lanes of a query are consecutive lanes of one warp: lane s of the
// query scans tile entries s, s + S, s + 2S, ...; every lane of the warp
// reaches the shuffles (no early exit).
template <int S>
__device__ __forceinline__ void combine_best(double& bd, int& bj) {
#pragma unroll
  for (int o = 1; o < S; o <<= 1) {
    const double d2 = __shfl_xor_sync(0xFFFFFFFFu, bd, o);
    const int j = __shfl_xor_sync(0xFFFFFFFFu, bj, o);
    take_best(bd, bj, d2, j);
  }
}

// Radius scan of one tile (entries s, s + S, ...): the FP32 box screen, then
// the exact FP64 test and the running strict minimum.
template <int S>
__device__ __forceinline__ void tile_radius(const Tile& T, const double* __restrict__ rx, const double* __restrict__ ry,
                                            int n, int s, int base, double xi, double yi, float xf, float yf, float Tf,
                                            double r2, int& c, double& bd, int& bj) {
#pragma unroll 4
  for (int t = s; t < n; t += S) {
    const float2 pf = T.f[t];
    const float dxf = xf - pf.x, dyf = yf - pf.y;
    if (fmaxf(fabsf(dxf), fabsf(dyf)) > Tf) continue;
    const double dx = xi - rx[base + t], dy = yi - ry[base + t];
    const double d2 = dx * dx + dy * dy;
    if (d2 <= r2) {
      ++c;
      if (bj < 0 || d2 < bd) {
        bd = d2;
        bj = base + t;
      }
    }
  }
}

// For each query point: number of reference points within eps (exact FP64
// test), and the nearest of them (strict <: the lowest index wins ties).
template <int S>
__global__ void __launch_bounds__(kBlock, 16) radius_best_kernel(int nq, const double* __restrict__ qx,
                                                              const double* __restrict__ qy, int nr,
                                                              const double* __restrict__ rx,
                                                              const double* __restrict__ ry,
                                                              const float2* __restrict__ rf, double r2, float T,
                                                              int* __restrict__ count, int* __restrict__ best_idx,
                                                              double* __restrict__ best_d2,
                                                              const GridHead* __restrict__ grid) {
  if (grid && grid->used()) return;  // searched through the grid
  __shared__ Tile tile;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int s = (int)(g % S);
  const long long i = g / S;
  const bool active = i < nq;
  const double xi = active ? qx[i] : 0.0, yi = active ? qy[i] : 0.0;
  const float xf = (float)xi, yf = (float)yi;
  int c = 0, bj = -1;
  double bd = 0.0;
  for (int base = 0; base < nr; base += kTile) {
    const int n = min(kTile, nr - base);
    __syncthreads();
    load_tile(tile, rf, base, n);
    __syncthreads();
    if (active) {
      if (n == kTile)
        tile_radius<S>(tile, rx, ry, kTile, s, base, xi, yi, xf, yf, T, r2, c, bd, bj);
      else
        tile_radius<S>(tile, rx, ry, n, s, base, xi, yi, xf, yf, T, r2, c, bd, bj);
    }
  }
#pragma unroll
  for (int o = 1; o < S; o <<= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
  combine_best<S>(bd, bj);
  if (active && s == 0) {
    count[i] = c;
    best_idx[i] = bj;
    best_d2[i] = bj < 0 ? 0.0 : bd;
  }
}

// Pass-1 screen of the nearest-neighbour search.  With D the smallest FP32
// distance d2_f of the query (pass 0), the true minimum is at most
// M = D + E(D), where E(x) = 2^-20 (x + R (sqrt(2x)/(1 - u) + 2^-62)) + R2c
// bounds e for any pair with d2_f = x (|dx_f| + |dy_f| <= sqrt(2 (dx_f^2 +
// dy_f^2)) <= sqrt(2 d2_f)/(1 - u), the 2^-62 covering FP32 underflow of the
// squares).  A point can be the exact minimiser only if d2_f - E(d2_f) <= M,
// i.e. sqrt(d2_f) <= (c1 + sqrt(c1^2 + 4a(c0 + M)))/(2a) with a = 1 - 2^-20,
// c1 = 2^-20 R sqrt2/(1 - u), c0 = 2^-82 R + R2c.  Everything is evaluated
// rounding upward (each quantity only grows), so the returned FP32 threshold
// admits every possible minimiser.
__device__ __forceinline__ float nearest_threshold(float D, double R, double R2c) {
  if (!(D < INFINITY)) return INFINITY;
  const double u1 = 1.0 / (1.0 - 0x1p-24) * (1.0 + 0x1p-50);  // >= 1/(1 - u)
  const double d = (double)D;
  const double c1 = __dmul_ru(__dmul_ru(0x1p-20 * R, 1.4142135623730952), u1);  // sqrt2 rounded up
  const double c0 = __dadd_ru(0x1p-82 * R, R2c);
  const double E = __dadd_ru(__dadd_ru(0x1p-20 * d, __dmul_ru(c1, __dsqrt_ru(d))), c0);
  const double M = __dadd_ru(d, E);
  const double a = 1.0 - 0x1p-20;
  const double disc = __dadd_ru(__dmul_ru(c1, c1), __dmul_ru(4.0 * a, __dadd_ru(c0, M)));
  const double smax = __ddiv_ru(__dadd_ru(c1, __dsqrt_ru(disc)), 2.0 * a);
  return __double2float_ru(__dmul_ru(smax, smax));
}

// Pass-0 scan of one tile: the smallest FP32 distance over entries s, s + S,
// ... (self excluded when the query's own index lies in the tile).
template <int S, bool SELF>
__device__ __forceinline__ float tile_min(const Tile& T, int cnt, int s, int self, float xf, float yf, float D) {
#pragma unroll 4
  for (int t = s; t < cnt; t += S) {
    if (SELF && t == self) continue;
    const float2 pf = T.f[t];
    const float dxf = xf - pf.x, dyf = yf - pf.y;
    D = fminf(D, __fadd_rn(__fmul_rn(dxf, dxf), __fmul_rn(dyf, dyf)));
  }
  return D;
}

// Pass-1 scan of one tile: exact FP64 distances of the entries under thr.
template <int S, bool SELF>
__device__ __forceinline__ void tile_best(const Tile& T, const double* __restrict__ px, const double* __restrict__ py,
                                          int cnt, int s, int self, int base, double xi, double yi, float xf, float yf,
                                          float thr, double& bd, int& bj) {
#pragma unroll 4
  for (int t = s; t < cnt; t += S) {
    const float2 pf = T.f[t];
    const float dxf = xf - pf.x, dyf = yf - pf.y;
    if (!(__fadd_rn(__fmul_rn(dxf, dxf), __fmul_rn(dyf, dyf)) <= thr) || (SELF && t == self)) continue;
    const double dx = xi - px[base + t], dy = yi - py[base + t];
    const double d2 = dx * dx + dy * dy;
    if (bj < 0 ? d2 < 1e300 : d2 < bd) {
      bd = d2;
      bj = base + t;
    }
  }
}

// Nearest neighbour of every point within its own set (excluding itself;
// strict <, the lowest index wins ties).  Pass 0 finds the smallest FP32
// distance, pass 1 decides in FP64 among the points under the threshold
// above, which contain every point whose true distance can be minimal.
// The query's own index is tested only in the tile that holds it; full tiles
// run a fixed trip count.
template <int S>
__global__ void __launch_bounds__(kBlock, 16) nearest_kernel(int n, const double* __restrict__ px,
                                                              const double* __restrict__ py,
                                                              const float2* __restrict__ pf, double R, double R2c,
                                                              int* __restrict__ out,
                                                              const GridHead* __restrict__ grid) {
  if (grid && grid->used()) return;  // searched through the grid
  __shared__ Tile tile;
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int s = (int)(g % S);
  const long long i = g / S;
  const bool active = i < n;
  const double xi = active ? px[i] : 0.0, yi = active ? py[i] : 0.0;
  const float xf = (float)xi, yf = (float)yi;
  float D = INFINITY;
  for (int base = 0; base < n; base += kTile) {
    const int cnt = min(kTile, n - base);
    __syncthreads();
    load_tile(tile, pf, base, cnt);
    __syncthreads();
    if (active) {
      const long long self = i - base;
      if (self >= 0 && self < cnt)
        D = tile_min<S, true>(tile, cnt, s, (int)self, xf, yf, D);
      else if (cnt == kTile)
        D = tile_min<S, false>(tile, kTile, s, -1, xf, yf, D);
      else
        D = tile_min<S, false>(tile, cnt, s, -1, xf, yf, D);
    }
  }
#pragma unroll
  for (int o = 1; o < S; o <<= 1) D = fminf(D, __shfl_xor_sync(0xFFFFFFFFu, D, o));
  const float thr = nearest_threshold(D, R, R2c);
  int bj = -1;
  double bd = 0.0;
  for (int base = 0; base < n; base += kTile) {
    const int cnt = min(kTile, n - base);
    __syncthreads();
    load_tile(tile, pf, base, cnt);
    __syncthreads();
    if (active) {
      const long long self = i - base;
      if (self >= 0 && self < cnt)
        tile_best<S, true>(tile, px, py, cnt, s, (int)self, base, xi, yi, xf, yf, thr, bd, bj);
      else if (cnt == kTile)
        tile_best<S, false>(tile, px, py, kTile, s, -1, base, xi, yi, xf, yf, thr, bd, bj);
      else
        tile_best<S, false>(tile, px, py, cnt, s, -1, base, xi, yi, xf, yf, thr, bd, bj);
    }
  }
  combine_best<S>(bd, bj);
  if (active && s == 0) out[i] = bj;
}

// ---------------------------------------------------------------------------
// Grid search.  Workspace of 8 n bytes: the points' indices sorted by cell
// (4 n), the cells' ends (4 G^2, G^2 <= n - 64), GridHead.  The cell of a
// coordinate is a monotone function of it (every rounding is), so all points
// with x in [a, b] lie in the cells cell(a) .. cell(b).
// ---------------------------------------------------------------------------
// Pairs above which the grid is built.  Building it takes 40 us, which a set that
// turns out too crowded for it pays beside the all-pairs scan (nearest: 8300
// points 260 -> 299 us, 24000 1397 -> 1436).  All pairs / grid, us, on a noisy
// curve and with a hundred points strewn around it:
//                8300               12000              16384
//   nearest   114 / 70, 115 / 122   177 / 78, 177 / 148   230 / 81, 229 / 193
//   radius     62 / 64,  60 / 77     87 / 68,  85 / 87    117 / 72, 119 / 95
constexpr long long kNearestPairs = 1ll << 26, kRadiusPairs = 1ll << 27;
constexpr int kGridMin = 4096;

__host__ __device__ inline int grid_side(int n) {
  const int most = n - 64 < (1 << 20) ? n - 64 : (1 << 20);
  int g = 1;
  while ((g + 1) * (g + 1) <= most) ++g;
  return g;
}

__device__ __forceinline__ unsigned long long order_key(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return (b >> 63) ? ~b : b | 0x8000000000000000ull;
}
__device__ __forceinline__ double key_value(unsigned long long k) {
  return __longlong_as_double((long long)((k >> 63) ? k & 0x7FFFFFFFFFFFFFFFull : ~k));
}
__device__ __forceinline__ int cell_of(double v, double v0, double inv, int G) {
  const double c = floor((v - v0) * inv);
  return c >= 1.0 ? (c < (double)G ? (int)c : G - 1) : 0;  // NaN: 0
}

__global__ void grid_init_kernel(int cells, int* __restrict__ ends, GridHead* __restrict__ h) {
  for (const int i : grid_strided(cells)) ends[i] = 0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    h->lo[0] = h->lo[1] = ~0ull;
    h->hi[0] = h->hi[1] = 0ull;
    h->work = 0;
    h->use = 0;
    h->far = 0;
  }
}

__global__ void __launch_bounds__(256) grid_box_kernel(int n, const double* __restrict__ x, const double* __restrict__ y,
                                                       GridHead* __restrict__ h) {
  unsigned long long lo[2] = {~0ull, ~0ull}, hi[2] = {0, 0};
  for (const int i : grid_strided(n)) {
    const unsigned long long k[2] = {order_key(x[i]), order_key(y[i])};
    for (int a = 0; a < 2; ++a) {
      lo[a] = min(lo[a], k[a]);
      hi[a] = max(hi[a], k[a]);
    }
  }
  for (int a = 0; a < 2; ++a) {
    for (int o = 16; o; o >>= 1) {
      lo[a] = min(lo[a], __shfl_xor_sync(0xFFFFFFFFu, lo[a], o));
      hi[a] = max(hi[a], __shfl_xor_sync(0xFFFFFFFFu, hi[a], o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&h->lo[a], lo[a]);
      atomicMax(&h->hi[a], hi[a]);
    }
  }
}

// Cell size: the larger extent over G cells, and at least `reach` (the radius
// search meets three by three cells).
__global__ void grid_size_kernel(int G, double reach, GridHead* __restrict__ h) {
  const double x0 = key_value(h->lo[0]), y0 = key_value(h->lo[1]);
  const double ex = key_value(h->hi[0]) - x0, ey = key_value(h->hi[1]) - y0;
  const double ext = fmax(ex, ey);
  const double cell = fmax(ext / (double)G, reach);
  const bool fine = ex >= 0.0 && ey >= 0.0 && ext < 1e150 && cell > 1e-150 && ext > 4.0 * reach;
  h->x0 = fine ? x0 : 0.0;
  h->y0 = fine ? y0 : 0.0;
  h->cell = fine ? cell : 1.0;
  h->inv = fine ? 1.0 / cell : 0.0;
  h->use = fine ? kUse : 0;
}

// Adds a warp's 32 points (cell -1: none) to their cells' numbers, one atomic a
// cell, and returns each point's own number: crowded points would otherwise
// queue one by one at their cell's address (65536 of them, twice: 0.9 ms).
__device__ __forceinline__ int add_to_cell(int* __restrict__ cells, int cell) {
  const int lane = threadIdx.x & 31;
  const unsigned same = __match_any_sync(0xFFFFFFFFu, cell);
  const int first = __ffs(same) - 1;
  int at = 0;
  if (lane == first && cell >= 0) at = atomicAdd(&cells[cell], __popc(same));
  return __shfl_sync(0xFFFFFFFFu, at, first) + __popc(same & ((1u << lane) - 1u));
}

// Calls f(i, cell) for every point, a warp's lanes together (i = n, cell -1 beyond).
template <class F>
__device__ __forceinline__ void each_cell(int n, const double* __restrict__ x, const double* __restrict__ y, int G,
                                          const GridHead* __restrict__ h, F f) {
  const int lane = threadIdx.x & 31;
  for (const int b : Strided{global_thread() - lane, (long long)gridDim.x * blockDim.x, n}) {
    const bool in = lane < n - b;
    const int i = in ? b + lane : n;
    f(i, in ? cell_of(y[i], h->y0, h->inv, G) * G + cell_of(x[i], h->x0, h->inv, G) : -1);
  }
}

__global__ void grid_count_kernel(int n, const double* __restrict__ x, const double* __restrict__ y, int G,
                                  const GridHead* __restrict__ h, int* __restrict__ counts) {
  if (!h->used()) return;
  each_cell(n, x, y, G, h, [&](int, int cell) { add_to_cell(counts, cell); });
}

// Candidates the queries meet in the three by three cells around them (the
// radius search's; nearly the nearest search's), from the cells' counts: a grid
// that is not worth using is neither scanned nor filled.
__global__ void __launch_bounds__(256) grid_work_kernel(int nq, const double* __restrict__ x,
                                                        const double* __restrict__ y, int G,
                                                        const int* __restrict__ counts, GridHead* __restrict__ h) {
  if (!h->used()) return;
  unsigned long long work = 0;
  for (const int i : grid_strided(nq)) {
    const int cx = cell_of(x[i], h->x0, h->inv, G), cy = cell_of(y[i], h->y0, h->inv, G);
    for (int r = max(cy - 1, 0); r <= min(cy + 1, G - 1); ++r)
      for (int c = max(cx - 1, 0); c <= min(cx + 1, G - 1); ++c) work += (unsigned)counts[r * G + c];
  }
  for (int o = 16; o; o >>= 1) work += __shfl_xor_sync(0xFFFFFFFFu, work, o);
  if ((threadIdx.x & 31) == 0) atomicAdd(&h->work, work);
}

// Counts to starts (one block; 16384 cells' loads in flight at once, scanned
// 4096 at a time), if the grid pays: while it meets at most a sixteenth of the
// pairs (a candidate costs several pairs of the all-pairs scan: two dependent
// loads).
__global__ void __launch_bounds__(1024) grid_scan_kernel(int cells, unsigned long long pairs, GridHead* __restrict__ h,
                                                         int* __restrict__ ends) {
  if (!h->used()) return;
  if (h->work > pairs / 16) {
    if (threadIdx.x == 0) h->use = 0;
    return;
  }
  constexpr int kRounds = 4;
  __shared__ int warp_sum[2][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int carry = 0, buf = 0;
  for (int base = 0; base < cells; base += 4096 * kRounds) {
    int v[kRounds][4];
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int at = base + 4096 * r + 4 * (int)threadIdx.x + e;
        v[r][e] = at < cells ? ends[at] : 0;
      }
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int sum = (v[r][0] + v[r][1]) + (v[r][2] + v[r][3]);
      int inc = sum;
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += u;
      }
      if (lane == 31) warp_sum[buf][w] = inc;
      __syncthreads();
      // every warp scans the warps' sums (two buffers in turn: one barrier a round)
      const int own = warp_sum[buf][lane];
      int t = own;
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xFFFFFFFFu, t, o);
        if (lane >= o) t += u;
      }
      int run = carry + __shfl_sync(0xFFFFFFFFu, t - own, w) + inc - sum;
      carry += __shfl_sync(0xFFFFFFFFu, t, 31);
      buf ^= 1;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int at = base + 4096 * r + 4 * (int)threadIdx.x + e;
        if (at < cells) ends[at] = run;
        run += v[r][e];
      }
    }
  }
}

// Points into their cells; the starts become the ends.
__global__ void grid_fill_kernel(int n, const double* __restrict__ x, const double* __restrict__ y, int G,
                                 const GridHead* __restrict__ h, int* __restrict__ ends, int* __restrict__ order) {
  if (!h->used()) return;
  each_cell(n, x, y, G, h, [&](int i, int cell) {
    const int at = add_to_cell(ends, cell);
    if (cell >= 0) order[at] = i;
  });
}

// Points of row cy, cells ca .. cb: order[first .. first + count).
__device__ __forceinline__ void row_range(const int* __restrict__ ends, int G, int cy, int ca, int cb, int& first,
                                          int& count) {
  const int c = cy * G + ca;
  first = c ? ends[c - 1] : 0;
  count = ends[cy * G + cb] - first;
}

// An FP32 value within 2^-23 |v| of v, 2^-126 where v is smaller than that, and
// the largest ones beyond FP32's range, on the integer pipe (a conversion holds
// the FP64 unit).
__device__ __forceinline__ float near_float(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const int e = (int)((hi & 0x7FF00000u) >> 20) - 1023 + 127;
  const unsigned m = ((hi & 0xFFFFFu) << 3) | (lo >> 29);
  const unsigned mag = e <= 0 ? 0u : (e >= 255 ? 0x7F7FFFFFu : ((unsigned)e << 23) | m);
  return __uint_as_float((hi & 0x80000000u) | mag);
}

// A candidate can matter only if |dx| and |dy| are at most `reach`; in FP32,
// with each coordinate within 2^-23 R (plus 2^-126) and the difference rounded,
// that is |dx_f|, |dy_f| <= (reach + 2^-21 R)(1 + 2^-20) + 2^-120.
__device__ __forceinline__ float screen_bound(double reach, double R) {
  return __double2float_ru(__dadd_ru(__dmul_ru(__dadd_ru(reach, 0x1p-21 * R), 1.0 + 0x1p-20), 0x1p-120));
}

// A warp's queries scan side by side; what passes the FP32 screen waits in a
// queue per lane, so that the FP64 decisions run on all lanes at once instead of
// whenever one of them has a pair.
// S lanes share a query's candidates (one / four lanes, us: 16384 points on a curve
// 103 / 72, with a hundred points around it 177 / 96).
constexpr int kRadiusQueue = 8;
template <int S>
__global__ void __launch_bounds__(128) radius_grid_kernel(int nq, const double* __restrict__ qx,
                                                          const double* __restrict__ qy, int G,
                                                          const double* __restrict__ rx,
                                                          const double* __restrict__ ry,
                                                          const int* __restrict__ ends, const int* __restrict__ order,
                                                          const GridHead* __restrict__ h, double eps, double reach,
                                                          double R, int* __restrict__ count,
                                                          int* __restrict__ best_idx, double* __restrict__ best_d2) {
  if (!h->used()) return;
  __shared__ int queue[kRadiusQueue][128];
  const int tx = threadIdx.x;
  const long long i = global_thread() / S;
  const int s = tx % S;
  const bool valid = i < nq;
  const double xi = valid ? qx[i] : 0.0, yi = valid ? qy[i] : 0.0, r2 = eps * eps;
  const float xf = near_float(xi), yf = near_float(yi), T = screen_bound(eps, R);
  int c = 0, bj = -1, queued = 0;
  double bd = 0.0;
  const int cl = cell_of(xi - reach, h->x0, h->inv, G), ch = cell_of(xi + reach, h->x0, h->inv, G);
  int row = cell_of(yi - reach, h->y0, h->inv, G);
  const int row_end = valid ? cell_of(yi + reach, h->y0, h->inv, G) : row - 1;
  int t = 0, left = 0;  // this lane's next candidate of the row, the row's from there on
  bool more = valid;
  auto skip = [&](int by) {
    const int taken = min(left, by);
    t += taken;
    left -= taken;
  };
  auto next_row = [&]() {
    row_range(ends, G, row, cl, ch, t, left);
    skip(4 * s);
  };
  if (valid) next_row();
  auto flush = [&]() {
    for (int e = 0; __any_sync(0xFFFFFFFFu, e < queued); ++e) {
      if (e >= queued) continue;
      const int j = queue[e][tx];
      const double dx = xi - rx[j], dy = yi - ry[j];
      const double d2 = dx * dx + dy * dy;
      if (d2 <= r2) {
        ++c;
        take_best(bd, bj, d2, j);
      }
    }
    queued = 0;
  };
  while (__any_sync(0xFFFFFFFFu, more)) {
    // four candidates of every lane's rows
    int j[4];
    double xj[4], yj[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) j[e] = e < left ? order[t + e] : -1;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      xj[e] = j[e] >= 0 ? rx[j[e]] : 0.0;
      yj[e] = j[e] >= 0 ? ry[j[e]] : 0.0;
    }
    if (__any_sync(0xFFFFFFFFu, queued > kRadiusQueue - 4)) flush();
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (j[e] >= 0 && !(fmaxf(fabsf(xf - near_float(xj[e])), fabsf(yf - near_float(yj[e]))) > T)) queue[queued++][tx] = j[e];
    skip(4 * S);
    while (more && left == 0) {
      if (++row > row_end)
        more = false;
      else
        next_row();
    }
  }
  flush();
  for (int o = 1; o < S; o <<= 1) {
    c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    const double d2 = __shfl_xor_sync(0xFFFFFFFFu, bd, o);
    const int j = __shfl_xor_sync(0xFFFFFFFFu, bj, o);
    take_best(bd, bj, d2, j);
  }
  if (!valid || s != 0) return;
  count[i] = c;
  best_idx[i] = bj;
  best_d2[i] = bj < 0 ? 0.0 : bd;
}

// The nearest point a query has met: the smallest squared distance below the
// all-pairs scan's first acceptance, ties to the smaller index.  FP32 distances
// decide while they can: a point is passed over when another one is certainly
// nearer, takes the place of one that is certainly farther, and only what lies in
// between is decided in FP64 (a search whose every improvement was, ln(c) a lane
// of c candidates, held the FP64 unit).
//
// With coordinates within 2^-23 R a distance f is off by at most a(f) = 2^-21.8 f
// + 2^-20.4 R sqrt(f) + 2^-43 R^2 (the header's derivation).  A point at g >
// f + E(f), E(f) = 2^-20 f + 2^-19 R sqrt(f) + 2^-38 R^2, is farther than one at f:
// g - a(g) grows from 2^-42.8 R^2 on, and at g = f + E(f) it exceeds f + a(f),
// as a(f) + a(f + E(f)) < E(f) (sqrt(f + E) <= sqrt(f) + sqrt(E)).  2^-120 more
// for squares below FP32's range; beyond it (R^2 infinite) E is infinite and every
// point is decided in FP64.
struct Nearest {
  double x, y;
  float xf, yf, R2, RR;
  float least, cut;  // FP32 distance of `at`; beyond `cut` a point is farther
  int at;            // nearest so far, not decided (-1: none)
  double bd;         // decided
  int bj;
  __device__ __forceinline__ Nearest(double px, double py, double R)
      : x(px), y(py), xf(near_float(px)), yf(near_float(py)), least(INFINITY), cut(INFINITY), at(-1), bd(1e300),
        bj(-1) {
    const float Rf = __double2float_ru(R);
    R2 = 2.0f * Rf;
    RR = fmaf(0x1p-38f * Rf, Rf, 0x1p-120f);
  }
  __device__ __forceinline__ float beyond(float d2) const {
    float s;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(s) : "f"(d2));
    return fmaf(0x1p-20f, fmaf(R2, s, d2), RR) + d2;
  }
  __device__ __forceinline__ void decide(double xj, double yj, int j) {
    const double dx = x - xj, dy = y - yj;
    const double d2 = dx * dx + dy * dy;
    if (d2 < bd || (d2 == bd && bj >= 0 && j < bj)) {
      bd = d2;
      bj = j;
    }
  }
  // a point decided elsewhere
  __device__ __forceinline__ void take(double d2, int j) {
    if (d2 < bd || (d2 == bd && (unsigned)j < (unsigned)bj)) {
      bd = d2;
      bj = j;
    }
  }
  __device__ __forceinline__ void settle(const double* px, const double* py) {
    if (at >= 0) decide(px[at], py[at], at);
    at = -1;
  }
  __device__ __forceinline__ float distance(float fx, float fy) const {
    const float dx = xf - fx, dy = yf - fy;
    return fmaf(dx, dx, dy * dy);
  }
  __device__ __forceinline__ void meet(double xj, double yj, int j, const double* px, const double* py) {
    const float d2 = distance(near_float(xj), near_float(yj));
    if (d2 > cut) return;
    const float c = d2 < least ? beyond(d2) : INFINITY;
    if (c < least) {  // nearer than any so far
      at = j;
      bd = 1e300;
      bj = -1;
    } else {
      settle(px, py);
      decide(xj, yj, j);
    }
    least = fminf(least, d2);
    cut = fminf(cut, c);
  }
};

// Nearest neighbours: a query (in cell order, so that a warp's meet the same
// cells) takes the three by three cells around its own, then ring after ring
// until the block's border is farther than the best found.  A query whose
// nearest point lies beyond kRings rings, or whose rings meet more than a 64th
// of all points, is left to nearest_far_kernel (kFar in `out`): its walk, two
// dependent loads a row and side and two for every four candidates, would go on
// alone, for up to G rings.
//
// S lanes share a query: the cells' candidates, or a ring's rows and sides.  The
// loads' latency bounds it, and far points make it longer: they widen the box and
// with it the cells (434 candidates a query of 65536 points on a noisy curve, 1432
// with a hundred points strewn around it).  Against one lane a query, every ring
// walked to its end and every improvement decided in FP64, ms: the curve 0.28 ->
// 0.18, with one far point 7.17 -> 0.28, with a hundred 2.13 -> 0.60; 16384 points
// 0.14 -> 0.08, 1.90 -> 0.11, 0.47 -> 0.19.
constexpr int kRings = 4;
constexpr int kFar = -2;
template <int S>
__global__ void __launch_bounds__(128) nearest_grid_kernel(int n, const double* __restrict__ x,
                                                           const double* __restrict__ y, int G,
                                                           const int* __restrict__ ends,
                                                           const int* __restrict__ order,
                                                           GridHead* __restrict__ h, double R,
                                                           int* __restrict__ out) {
  if (!h->used()) return;
  const long long q = global_thread() / S;
  if (q >= n) return;
  const int s = threadIdx.x % S;
  const unsigned group = ((1u << S) - 1u) << ((threadIdx.x & 31) - s);
  const int i = order[q];
  Nearest best(x[i], y[i], R);
  const double x0 = h->x0, y0 = h->y0, cell = h->cell;
  const int cx = cell_of(best.x, x0, h->inv, G), cy = cell_of(best.y, y0, h->inv, G);
  int budget = INT_MAX;  // candidates this lane may still meet; below zero: too many
  // row r's cells ca .. cb; `part` of the row's `parts` lanes
  auto visit = [&](int r, int ca, int cb, int part, int parts) {
    if (r < 0 || r >= G || cb < 0 || ca >= G || budget < 0) return;
    int a, c;
    row_range(ends, G, r, max(ca, 0), min(cb, G - 1), a, c);
    budget = c > budget ? -1 : budget - c;
    if (budget < 0) return;
    for (int t = 4 * part; t < c; t += 4 * parts) {
      int j[4];
      double xj[4], yj[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) j[e] = order[a + min(t + e, c - 1)];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        xj[e] = x[j[e]];
        yj[e] = y[j[e]];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e)  // (a repeated last candidate changes nothing)
        if (j[e] != i) best.meet(xj[e], yj[e], j[e], x, y);
    }
  };
  // what the lanes found, in each of them
  auto share = [&]() {
    best.settle(x, y);
    for (int o = 1; o < S; o <<= 1) {
      const double d2 = __shfl_xor_sync(group, best.bd, o);
      const int j = __shfl_xor_sync(group, best.bj, o);
      best.least = fminf(best.least, __shfl_xor_sync(group, best.least, o));
      best.cut = fminf(best.cut, __shfl_xor_sync(group, best.cut, o));
      budget = min(budget, __shfl_xor_sync(group, budget, o));
      best.take(d2, j);
    }
  };
  // (its own row first: what it finds there rules out most of the others')
  visit(cy, cx - 1, cx + 1, s, S);
  visit(cy - 1, cx - 1, cx + 1, s, S);
  visit(cy + 1, cx - 1, cx + 1, s, S);
  budget = n / 64;
  for (int k = 1;; ++k) {
    share();
    // every point outside the block of radius k is at least this far away (the
    // cells' borders are off by their rounding)
    double far = INFINITY;
    if (cx - k > 0) far = fmin(far, best.x - (x0 + (double)(cx - k) * cell));
    if (cx + k + 1 < G) far = fmin(far, (x0 + (double)(cx + k + 1) * cell) - best.x);
    if (cy - k > 0) far = fmin(far, best.y - (y0 + (double)(cy - k) * cell));
    if (cy + k + 1 < G) far = fmin(far, (y0 + (double)(cy + k + 1) * cell) - best.y);
    if (budget >= 0) {
      if (!(far < INFINITY)) break;  // the block covers the grid
      far = far * (1.0 - 0x1p-40) - 0x1p-40 * (R + cell);
      if (far > 0.0 && far * far * (1.0 - 0x1p-40) > best.bd) break;
    }
    if (k > kRings || budget < 0) {
      best.bj = kFar;
      h->far = 1;
      break;
    }
    // the ring: two rows, then 2 k + 1 cells of each side
    for (int u = s; u < 4 * k + 4; u += S) {
      const int v = u - 2, side = (v & 1) ? cx + k + 1 : cx - k - 1;
      if (v < 0)
        visit(u == 0 ? cy - k - 1 : cy + k + 1, cx - k - 1, cx + k + 1, 0, 1);
      else
        visit(cy - k + (v >> 1), side, side, 0, 1);
    }
  }
  if (s == 0) out[i] = best.bj;
}

// The queries nearest_grid_kernel left, a block each, over all points.  Either
// they lie five cells from any other point, so with no more cells than points
// there are at most about n / 16 of them; or a cell or more from any other, within
// five of a 64th of all points, which leaves room for a few thousand.  A block's
// share is strided: far points tend to follow each other.  Two passes, as the
// all-pairs scan: the block's least FP32 distance, then what it does not rule out.
constexpr int kFarBlock = 512, kFarTile = 8 * kFarBlock;
__global__ void __launch_bounds__(kFarBlock) nearest_far_kernel(int n, const double* __restrict__ x,
                                                                const double* __restrict__ y,
                                                                const float2* __restrict__ pf,
                                                                const GridHead* __restrict__ h, double R,
                                                                int* __restrict__ out) {
  if (!h->used() || !h->far) return;
  __shared__ int list[kFarBlock], listed;
  __shared__ double warp_d[kFarBlock / 32];
  __shared__ int warp_j[kFarBlock / 32];
  __shared__ float warp_least[kFarBlock / 32];
  const int tx = threadIdx.x;
  const unsigned keep = n - kHeadPoints, tiles = keep / kFarTile;
  for (long long base = 0; blockIdx.x + base * gridDim.x < n; base += kFarBlock) {
    const long long q = blockIdx.x + (base + tx) * gridDim.x;
    const bool far = q < n && out[q] == kFar;
    if (tx == 0) listed = 0;
    if (!__syncthreads_or(far)) continue;
    if (far) list[atomicAdd(&listed, 1)] = (int)q;
    __syncthreads();
    const int m = listed;
    for (int u = 0; u < m; ++u) {
      const int i = list[u];
      Nearest best(x[i], y[i], R);
      // FP32 distances of this thread's points (as many iterations in every thread)
      auto scan = [&](auto meet) {
        unsigned b = tx;
        for (unsigned t = 0; t < tiles; ++t, b += kFarTile) {
          float2 f[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = pf[b + e * kFarBlock];
#pragma unroll
          for (int e = 0; e < 8; ++e) meet(best.distance(f[e].x, f[e].y), b + e * kFarBlock);
        }
        for (; b < (unsigned)n; b += kFarBlock) {
          const float2 f = b < keep ? pf[b] : make_float2((float)x[b], (float)y[b]);
          meet(best.distance(f.x, f.y), b);
        }
      };
      float least = INFINITY;
      scan([&](float d2, unsigned j) { least = fminf(least, j == (unsigned)i ? INFINITY : d2); });
      least = __uint_as_float(__reduce_min_sync(0xFFFFFFFFu, __float_as_uint(least)));
      if ((tx & 31) == 0) warp_least[tx >> 5] = least;
      __syncthreads();
      least = __uint_as_float(
          __reduce_min_sync(0xFFFFFFFFu, __float_as_uint(warp_least[(tx & 31) % (kFarBlock / 32)])));
      const float cut = best.beyond(least);
      scan([&](float d2, unsigned j) {
        if (!(d2 > cut) && j != (unsigned)i) best.decide(x[j], y[j], (int)j);
      });
      auto over_warp = [&]() {
        for (int o = 16; o; o >>= 1) {
          const double d2 = __shfl_xor_sync(0xFFFFFFFFu, best.bd, o);
          const int j = __shfl_xor_sync(0xFFFFFFFFu, best.bj, o);
          best.take(d2, j);
        }
      };
      over_warp();
      if ((tx & 31) == 0) {
        warp_d[tx >> 5] = best.bd;
        warp_j[tx >> 5] = best.bj;
      }
      __syncthreads();
      if (tx < 32) {
        best.bd = warp_d[tx % (kFarBlock / 32)];
        best.bj = warp_j[tx % (kFarBlock / 32)];
        over_warp();
        if (tx == 0) out[i] = best.bj;
      }
      __syncthreads();
    }
  }
}

// Builds the grid of n reference points in ws and decides whether the nq
// queries use it; `reach`: the least cell size.
GridHead* build_grid(int nq, const double* qx, const double* qy, int n, const double* x, const double* y, double reach,
                     void* ws, int** ends, int** order, int* side, cudaStream_t st) {
  const int G = grid_side(n), cells = G * G;
  *order = (int*)ws;
  *ends = *order + n;
  *side = G;
  GridHead* h = (GridHead*)((char*)ws + 8 * (long long)n - 256);
  const unsigned blocks = std::min(blocks_of(n, 256), 1216u);
  grid_init_kernel<<<blocks, 256, 0, st>>>(cells, *ends, h);
  grid_box_kernel<<<blocks, 256, 0, st>>>(n, x, y, h);
  grid_size_kernel<<<1, 1, 0, st>>>(G, reach, h);
  grid_count_kernel<<<blocks, 256, 0, st>>>(n, x, y, G, h, *ends);
  grid_work_kernel<<<std::min(blocks_of(nq, 256), 1216u), 256, 0, st>>>(nq, qx, qy, G, *ends, h);
  grid_scan_kernel<<<1, 1024, 0, st>>>(cells, (unsigned long long)nq * (unsigned long long)n, h, *ends);
  grid_fill_kernel<<<blocks, 256, 0, st>>>(n, x, y, G, h, *ends, *order);
  return h;
}
bool grid_worth(long long nq, long long n, long long pairs) { return n >= kGridMin && nq * n > pairs; }

// Lanes per query: the largest of `most`, most / 2, ... 1 whose grid still fits in
// one wave of resident blocks (more lanes per query shorten each lane's scan;
// a second partial wave would cost a whole extra scan).
template <class K>
int lanes_per_query(K kernel, long long n, int block = kBlock, int most = 8) {
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0) != cudaSuccess)
    return 1;
  const long long resident = (long long)sms * per_sm * block;
  for (int S = most; S > 1; S >>= 1)
    if (n * S <= resident) return S;
  return 1;
}

int check(const char* what) {
  (void)what;
  return cudaGetLastError() == cudaSuccess ? HG_OK : HG_ERR_CUDA;
}

// Segment refinement of the connection pairs (connections/backends.py:237-320,
// _closest_points_on_segments_2d, and the interpolation of :480-520): pair k
// joins a0 = pu[I], a1 = pu[IU] with b0 = ps[J], b1 = ps[JS]; where ok[k] its
// closest-point parameters s, t (the reference's scalar arithmetic and
// clamping order, every product and sum rounded on its own) give the states
// (1 - s) Xu[I] + s Xu[IU], (1 - t) Xs[J] + t Xs[JS] and the midpoint of the
// two closest points; elsewhere Xu[I], Xs[J] and pu[I].  An index outside its
// set writes NaN (it cannot come from the searches).
__global__ void refine_pairs_kernel(int n, const int* __restrict__ I, const int* __restrict__ IU,
                                    const int* __restrict__ J, const int* __restrict__ JS,
                                    const unsigned char* __restrict__ ok, int nu, const double* __restrict__ pu,
                                    const double* __restrict__ Xu, int ns, const double* __restrict__ ps,
                                    const double* __restrict__ Xs, double* __restrict__ xu, double* __restrict__ xs,
                                    double* __restrict__ pt) {
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = I[k], j = J[k];
    const bool use = ok[k] != 0;
    const int iu = use ? IU[k] : i, js = use ? JS[k] : j;
    if (i < 0 || i >= nu || iu < 0 || iu >= nu || j < 0 || j >= ns || js < 0 || js >= ns) {
      for (int c = 0; c < 6; ++c) xu[6 * k + c] = xs[6 * k + c] = nan("");
      pt[2 * k] = pt[2 * k + 1] = nan("");
      continue;
    }
    if (!use) {
      for (int c = 0; c < 6; ++c) {
        xu[6 * k + c] = Xu[6LL * i + c];
        xs[6 * k + c] = Xs[6LL * j + c];
      }
      pt[2 * k] = pu[2LL * i];
      pt[2 * k + 1] = pu[2LL * i + 1];
      continue;
    }
    const double a0x = pu[2LL * i], a0y = pu[2LL * i + 1], a1x = pu[2LL * iu], a1y = pu[2LL * iu + 1];
    const double b0x = ps[2LL * j], b0y = ps[2LL * j + 1], b1x = ps[2LL * js], b1y = ps[2LL * js + 1];
    const double ux = a1x - a0x, uy = a1y - a0y, vx = b1x - b0x, vy = b1y - b0y;
    const double wx = a0x - b0x, wy = a0y - b0y;
    const double A = ux * ux + uy * uy, B = ux * vx + uy * vy, Cc = vx * vx + vy * vy;
    const double D = ux * wx + uy * wy, E = vx * wx + vy * wy;
    const double den = A * Cc - B * B;
    double s = 0.0, t = 0.0;
    if (den > 0.0) {
      s = (B * E - Cc * D) / den;
      t = (A * E - B * D) / den;
    }
    if (s < 0.0) {
      s = 0.0;
      if (Cc > 0.0) t = E / Cc;
    } else if (s > 1.0) {
      s = 1.0;
      if (Cc > 0.0) t = (E + B) / Cc;
    }
    if (t < 0.0) {
      t = 0.0;
      if (A > 0.0) {
        s = -D / A;
        s = s < 0.0 ? 0.0 : (s > 1.0 ? 1.0 : s);
      }
    } else if (t > 1.0) {
      t = 1.0;
      if (A > 0.0) {
        s = (B - D) / A;
        s = s < 0.0 ? 0.0 : (s > 1.0 ? 1.0 : s);
      }
    }
    for (int c = 0; c < 6; ++c) {
      xu[6 * k + c] = (1.0 - s) * Xu[6LL * i + c] + s * Xu[6LL * iu + c];
      xs[6 * k + c] = (1.0 - t) * Xs[6LL * j + c] + t * Xs[6LL * js + c];
    }
    pt[2 * k] = 0.5 * ((a0x + s * ux) + (b0x + t * vx));
    pt[2 * k + 1] = 0.5 * ((a0y + s * uy) + (b0y + t * vy));
  }
}

long long points_ws_bytes(long long n) { return ((n * (long long)sizeof(float2)) + 255) & ~255LL; }

// Workspace of a point set: the caller's when one is given (*owned = false),
// else stream-ordered scratch that the caller frees on the stream after the
// search (*owned = true); nullptr on failure.
void* points_ws(int n, void* ws, long long ws_bytes, bool* owned, cudaStream_t st) {
  void* p = ws;
  *owned = false;
  if (p) {
    if (ws_bytes < points_ws_bytes(n) || ((uintptr_t)p & 15) != 0) return nullptr;
  } else {
    if (cudaMallocAsync(&p, (size_t)n * sizeof(float2), st) != cudaSuccess) return nullptr;
    *owned = true;
  }
  return p;
}

// FP32 copy of a point set in its workspace (left out where the grid, whose
// storage it takes, answered every query).
void float2_copy(int n, const double* x, const double* y, float2* out, const GridHead* grid, cudaStream_t st) {
  const int blocks = (int)std::min<long long>(((long long)n + 255) / 256, 4096);
  to_float2_kernel<<<blocks, 256, 0, st>>>(n, x, y, out, grid);
}

}  // namespace

extern "C" {

long long hg_points_workspace_bytes(int n) { return n < 0 ? -1 : points_ws_bytes(n); }

int hg_radius_best(int nq, const double* qx, const double* qy, int nr, const double* rx, const double* ry, double eps,
                   double coord_max, int* count, int* best_idx, double* best_d2, void* workspace,
                   long long workspace_bytes, void* stream) {
  if (nq < 0 || nr < 0 || !(eps >= 0.0) || !(coord_max >= 0.0)) return HG_ERR_ARGS;
  if (workspace && (workspace_bytes < points_ws_bytes(nr) || ((uintptr_t)workspace & 15) != 0)) return HG_ERR_ARGS;
  if (nq == 0) return HG_OK;
  if (!qx || !qy || !count || !best_idx || !best_d2 || (nr > 0 && (!rx || !ry))) return HG_ERR_ARGS;
  const double T = (eps + 0x1p-22 * coord_max) * (1.0 + 0x1p-20);
  const float Tf = nextafterf((float)T, INFINITY);
  const cudaStream_t st = (cudaStream_t)stream;
  bool owned = false;
  float2* rf = nr > 0 ? (float2*)points_ws(nr, workspace, workspace_bytes, &owned, st) : nullptr;
  if (nr > 0 && !rf) return HG_ERR_CUDA;
  GridHead* grid = nullptr;
  if (grid_worth(nq, nr, kRadiusPairs)) {
    int *ends, *order, G;
    // past the rounding of the query's own coordinate and of the pair test
    const double reach = eps * (1.0 + 0x1p-40) + 0x1p-40 * coord_max;
    grid = build_grid(nq, qx, qy, nr, rx, ry, reach, rf, &ends, &order, &G, st);
    auto kernel = radius_grid_kernel<1>;
    const int S = lanes_per_query(radius_grid_kernel<4>, nq, 128, 4);
    if (S == 2) kernel = radius_grid_kernel<2>;
    if (S == 4) kernel = radius_grid_kernel<4>;
    kernel<<<blocks_of((long long)nq * S, 128), 128, 0, st>>>(nq, qx, qy, G, rx, ry, ends, order, grid, eps, reach,
                                                              coord_max, count, best_idx, best_d2);
  }
  if (nr > 0) float2_copy(nr, rx, ry, rf, grid, st);
  const int S = lanes_per_query(radius_best_kernel<8>, nq);
  const long long blocks = ((long long)nq * S + kBlock - 1) / kBlock;
  if (S == 8)
    radius_best_kernel<8><<<(unsigned)blocks, kBlock, 0, st>>>(nq, qx, qy, nr, rx, ry, rf, eps * eps, Tf, count, best_idx, best_d2, grid);
  else if (S == 4)
    radius_best_kernel<4><<<(unsigned)blocks, kBlock, 0, st>>>(nq, qx, qy, nr, rx, ry, rf, eps * eps, Tf, count, best_idx, best_d2, grid);
  else if (S == 2)
    radius_best_kernel<2><<<(unsigned)blocks, kBlock, 0, st>>>(nq, qx, qy, nr, rx, ry, rf, eps * eps, Tf, count, best_idx, best_d2, grid);
  else
    radius_best_kernel<1><<<(unsigned)blocks, kBlock, 0, st>>>(nq, qx, qy, nr, rx, ry, rf, eps * eps, Tf, count, best_idx, best_d2, grid);
  if (owned) cudaFreeAsync(rf, st);
  return check("radius_best_kernel");
}

int hg_nearest_neighbor(int n, const double* x, const double* y, double coord_max, int* out, void* workspace,
                        long long workspace_bytes, void* stream) {
  if (n < 0 || !(coord_max >= 0.0)) return HG_ERR_ARGS;
  if (workspace && (workspace_bytes < points_ws_bytes(n) || ((uintptr_t)workspace & 15) != 0)) return HG_ERR_ARGS;
  if (n == 0) return HG_OK;
  if (!x || !y || !out) return HG_ERR_ARGS;
  // R and 2^-43 R^2 as FP32 values rounded up (the bound's constants), passed in FP64
  const double R = (double)nextafterf((float)coord_max, INFINITY);
  const double R2c = (double)nextafterf((float)(0x1p-43 * coord_max * coord_max), INFINITY);
  const cudaStream_t st = (cudaStream_t)stream;
  bool owned = false;
  float2* pf = (float2*)points_ws(n, workspace, workspace_bytes, &owned, st);
  if (!pf) return HG_ERR_CUDA;
  GridHead* grid = nullptr;
  if (grid_worth(n, n, kNearestPairs)) {
    int *ends, *order, G;
    grid = build_grid(n, x, y, n, x, y, 0.0, pf, &ends, &order, &G, st);
    const int S = lanes_per_query(nearest_grid_kernel<4>, n, 128, 4);
    auto kernel = nearest_grid_kernel<1>;
    if (S == 2) kernel = nearest_grid_kernel<2>;
    if (S == 4) kernel = nearest_grid_kernel<4>;
    kernel<<<blocks_of((long long)n * S, 128), 128, 0, st>>>(n, x, y, G, ends, order, grid, coord_max, out);
  }
  float2_copy(n, x, y, pf, grid, st);
  if (grid) nearest_far_kernel<<<304, kFarBlock, 0, st>>>(n, x, y, pf, grid, coord_max, out);
  const int S = lanes_per_query(nearest_kernel<8>, n);
  const long long blocks = ((long long)n * S + kBlock - 1) / kBlock;
  if (S == 8)
    nearest_kernel<8><<<(unsigned)blocks, kBlock, 0, st>>>(n, x, y, pf, R, R2c, out, grid);
  else if (S == 4)
    nearest_kernel<4><<<(unsigned)blocks, kBlock, 0, st>>>(n, x, y, pf, R, R2c, out, grid);
  else if (S == 2)
    nearest_kernel<2><<<(unsigned)blocks, kBlock, 0, st>>>(n, x, y, pf, R, R2c, out, grid);
  else
    nearest_kernel<1><<<(unsigned)blocks, kBlock, 0, st>>>(n, x, y, pf, R, R2c, out, grid);
  if (owned) cudaFreeAsync(pf, st);
  return check("nearest_kernel");
}

int hg_connection_refine(int n, const int* I, const int* IU, const int* J, const int* JS, const unsigned char* ok,
                         int nu, const double* pu, const double* Xu, int ns, const double* ps, const double* Xs,
                         double* xu, double* xs, double* pt, void* stream) {
  if (n < 0 || nu < 0 || ns < 0) return HG_ERR_ARGS;
  if (n == 0) return HG_OK;
  if (!I || !IU || !J || !JS || !ok || !pu || !Xu || !ps || !Xs || !xu || !xs || !pt) return HG_ERR_ARGS;
  const int blocks = (int)std::min<long long>(((long long)n + 127) / 128, 4096);
  refine_pairs_kernel<<<blocks, 128, 0, (cudaStream_t)stream>>>(n, I, IU, J, JS, ok, nu, pu, Xu, ns, ps, Xs, xu, xs,
                                                                 pt);
  return check("refine_pairs_kernel");
}

}  // extern "C"
