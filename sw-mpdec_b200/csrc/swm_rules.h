// swm_rules.h -- rules of the solvers' control flow as plain functions, for device and
// host code alike (a host compiler builds them as they are for the tests).
#pragma once

#ifdef __CUDACC__
#define SWM_HD __host__ __device__ __forceinline__
#else
#define SWM_HD inline
#endif

namespace swm {

// A grid barrier's arrival count has reached the target of its n-th use, n times the
// blocks.  Both grow by one per arrival modulo 2^32 and are never further apart than the
// blocks of a grid (no block arrives at a use before all have arrived at the one before
// it), so the sign of their difference tells, also where they pass 2^32.
SWM_HD bool barrier_open(unsigned int count, unsigned int target) {
  return (int)(count - target) >= 0;
}

// Position `steps` (0..n) after `pos` (0..n-1) in a ring of n.  The passes of a step can
// be more than an int counts (13 solves of any jacobi_maxiter), so positions are kept,
// not pass numbers.
SWM_HD int ring_at(int pos, int steps, int n) {
  const int p = pos + steps;
  return p >= n ? p - n : p;
}

// Half width, relative to the threshold, of the band of FP64 residual sums that leave the
// decision to exact sums.
constexpr double kBand = 0x1p-20;

// A pass's sum s of n terms, in any order, against the stop threshold: 1 stop, 0 go on, -1
// inside the band (NaN and infinite sums go on, as in exact sums).  n 2^-100 covers the
// truncation of the exact rule's terms; kBand the rounding of s (within n 2^-53 < 2^-24)
// and of thresh, the double nearest the limbs (limbs_value: within 2^-51).
SWM_HD int stop_decision(double s, double thresh, double n) {
  const double slack = n * 0x1p-100;
  if (!(s <= thresh * (1.0 + kBand) + slack)) return 0;
  return s <= thresh * (1.0 - kBand) - slack ? 1 : -1;
}

// Whether the RHS leaves its mass fluxes over dx, dy: only the exact assembly (time schemes
// 5 to 7, not the fast forms) reads the quotients.
SWM_HD bool fluxes_over_len(int timescheme, bool fast) { return timescheme > 4 && !fast; }

// The fastest of n schedules, tried in order: form(i) is 0 or 1, time(i) its time, negative
// when it failed (which ends the search: -1).  A form whose first schedule takes a fifth
// longer than the best so far is not tried further; a later schedule of a form says
// nothing about the others.
template <typename Form, typename Time>
inline int fastest_schedule(int n, Form form, Time time) {
  int pick = -1;
  float best = 0.f;
  bool tried[2] = {}, skip[2] = {};
  for (int i = 0; i < n; ++i) {
    const int f = form(i);
    if (skip[f]) continue;
    const float ms = time(i);
    if (ms < 0.f) return -1;
    if (!tried[f] && pick >= 0 && ms > 1.2f * best) skip[f] = true;
    tried[f] = true;
    if (pick < 0 || ms < best) {
      best = ms;
      pick = i;
    }
  }
  return pick;
}

}  // namespace swm
