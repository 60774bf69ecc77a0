// Library-internal functions shared between translation units; not part of
// the C ABI (include/hitengpu.h).
#pragma once

#include "hitengpu.h"

namespace hg_internal {

// The handle's grow-only device buffer of hg_correct_halo: at least `bytes`
// (allocated, and counted, only when the buffer is smaller).
int correct_buffers(hg_handle* h, long long bytes, void** out);
// hg_reserve from inside the library.
int reserve_refine(hg_handle* h, int N, int dim, int max_hits);
// Record `msg` as the handle's last error and return `code`.
int fail_msg(hg_handle* h, int code, const char* msg);
// The handle's slot for the device corrector's cached graph; free_fn
// releases it when the handle is destroyed.
void** graph_slot(hg_handle* h, void (*free_fn)(void*));
// Add n to the handle's kernel-launch counter.
void count_launches(hg_handle* h, long long n);
// The handle's device ordinal and a tuning value (hg_set_tuning keys).
int device_of(const hg_handle* h);
int tuning(const hg_handle* h, int key);

// Lanes per 6-dim trajectory for a launch that steps n of them side by side:
// the layout with the least time per step (30: five six-lane groups on one
// trajectory, a warp each).  A layout's step takes its latency while its warps
// fit an SM's FP64 unit (`cap` of them; in between the fourth-power mean of
// both fits the measurements within 6 %) and grows with the warps per SM
// beyond.  Measured on GB300 (us per DOP853 step, 152 SMs):
//   n         1     608    912    1216   3040   4864   7296   9728   14592  19456  29184  48640
//   1 lane    55.0  55.3   55.2   55.2   55.2   55.2   55.2   55.3   55.3   56.5   71.4   114
//   2 lanes   31.8  35.0   35.0   35.0   35.0   35.1   35.2   35.8   41.6   50.0   97.5   140
//   6 lanes   17.4  18.7   18.7   18.6   19.4   25.4   34.8   45.9   70.4   92.6   132    211
//   30 lanes  15.1  16.1   17.4   21.2   (57 at 2280)
// sm_capacity (the tuning value, 3 by default) moves the capacities.
inline int lanes_d6(long long n, int sms, double sm_capacity) {
  const int gs[4] = {30, 6, 2, 1};
  const long long per_warp[4] = {1, 5, 16, 32};
  const double lat[4] = {0.287, 0.337, 0.634, 1.0}, cap[4] = {6.6, 5.15, 6.03, 5.07};
  int best = 1;
  double best_cost = 0.0;
  for (int i = 0; i < 4; ++i) {
    const double warps = (double)((n + per_warp[i] - 1) / per_warp[i]);
    const double slots = (cap[i] + 0.5 * (sm_capacity - 3.0)) * sms;
    const double l2 = (warps / slots) * (warps / slots), lat2 = lat[i] * lat[i];
    const double cost = lat2 * lat2 * (1.0 + l2 * l2);
    if (i == 0 || cost < best_cost) {
      best = gs[i];
      best_cost = cost;
    }
  }
  return best;
}

// Layout of an event-free single-pass 42-dim run of n trajectories: 18 (three
// warps per five of them, four for DOP853) while an SM holds at most three such
// groups, warp pairs (12) beyond.  Measured on GB300 (us per step; G = 7 and 14
// are behind at every size):
//   n               760    1024   1500   2048   4096   8192
//   RK8, 18         26.9   30.6   30.6   41.2   76.4   140
//   RK8, pair       41.4   41.7   41.6   44.1   72.5   159
//   DOP853, 18      34.1   40.6   40.5   53.1   104    204
//   DOP853, pair    51.7   52.1   52.2   55.9   90.2   178
inline int lanes_d42_free(long long n, int sms, double sm_capacity) {
  const double groups = (double)((n + 4) / 5);
  return groups <= sm_capacity * sms ? 18 : 12;
}

// Lanes per crossing of a deferred refinement of up to `records` 6-dim
// crossings.  Six lanes halve the latency (a component of the dense cache a
// lane, two halvings a pass), one lane takes fewer FP64 instructions a
// crossing.  Measured on GB300 (us, 152 SMs; the lines meet at 43 an SM):
//   records    50    400   1237   2500   4000   6000   8000   16384
//   one lane   82.8  74.7  74.6   74.3   74.0   74.6   74.7   80.7
//   six lanes  33.5  34.1  34.8   38.2   52.4   66.8   90.0   183
inline int refine_lanes(long long records, int sms) { return records <= 40LL * sms ? 6 : 1; }

}  // namespace hg_internal
