// photic_starts.cuh -- a pixel's depth starts run as work items of their
// own and compared afterwards, for the kernels that give a pixel to a warp
// or a group of lanes (photic_region.cu, photic_joint_group.cu).
//
// samodel_optimise_one_bottom_combination runs the starts in sequence, keeps
// the best and ends at the first improvement below the early-exit cost
// (model/samodel.c:2380-2405).  The starts do not depend on one another, so
// they are queue positions (the first starts of all pixels, then the second,
// ...); each leaves a record, and the item that completes the starts up to
// the early exit (or all of them) compares the records in the order of the
// starts, which gives the sequential loop's result.  An item whose pixel has
// met the exit at an earlier start is dropped.
#pragma once
#include <stdint.h>

#include "photic_kernels.h"
#include "photic_softfp.cuh"

namespace photic {

// Publish start k's completion (its record is written); true for the one
// caller that is to compare the pixel's records.  One lane's part of the next.
__device__ __forceinline__ bool start_done_lane(const StartWork &w, int64_t slot, int k,
                                                int n_starts, double y, double early) {
  if (sf::lt(y, early) && sf::lt(y, 1.0e4)) atomicMin(w.exit_k + slot, k);
  __threadfence();
  const unsigned long long bit = 1ull << k;
  const unsigned long long mask = atomicOr(w.done + slot, bit) | bit;
  __threadfence();
  const int ex = __ldcg(w.exit_k + slot);
  const int last = ex < n_starts - 1 ? ex : n_starts - 1;
  const unsigned long long needed = (2ull << last) - 1;  // n_starts <= 32
  if ((mask & needed) != needed || (mask >> 63)) return false;
  const bool mine = !(atomicOr(w.done + slot, 1ull << 63) >> 63);
  if (mine) __threadfence();
  return mine;
}

// The same for the `width` lanes of `mask`, of which gl is the caller's rank
// and which have written the record between them: one answer.  The lanes that
// then read the other starts' records are behind the first lane's look at who
// has written them by the second barrier; exchanges order no memory.
__device__ __forceinline__ bool start_done(const StartWork &w, int64_t slot, int k, int n_starts,
                                           double y, double early, unsigned mask, int width,
                                           int gl) {
  __threadfence();
  __syncwarp(mask);
  int mine = 0;
  if (gl == 0) mine = start_done_lane(w, slot, k, n_starts, y, early);
  mine = __shfl_sync(mask, mine, 0, width);
  __syncwarp(mask);
  return mine != 0;
}

// Whether start k of the pixel whose word is *exit_k is still wanted: one
// answer for the `width` lanes of `mask`, of which gl is the caller's rank.
// Other warps lower the word meanwhile, so lanes that each loaded it could
// disagree, and the exchanges and barriers that follow would then be met by a
// part of the group: the first lane reads it and hands the rest its word.
__device__ __forceinline__ bool start_wanted(const int32_t *exit_k, int k, unsigned mask, int width,
                                             int gl) {
  int32_t ex = 0;
  if (gl == 0) ex = __ldcg(exit_k);
  return __shfl_sync(mask, ex, 0, width) >= k;
}

struct StartChoice {
  int32_t total, kept_evals, kept_start, kept_fault;
  bool invalid;  // a start hit the defensive evaluation cap
};

// The records compared as the sequential loop does; kept_start is -1 when no
// start got below the initial 1e4.
__device__ __forceinline__ StartChoice choose_start(const StartWork &w, int64_t slot, int n_starts,
                                                    double early) {
  StartChoice c = {0, 0, -1, 0, false};
  double lowest = 1.0e4;
#pragma unroll 1
  for (int k = 0; k < n_starts; k++) {
    const int64_t i = slot * n_starts + k;
    const int32_t ev = __ldcg(w.evals + i);
    if (ev < 0) {
      c.invalid = true;
      break;
    }
    c.total += ev;
    const double y = __ldcg(w.y + i);
    if (sf::lt(y, lowest)) {
      lowest = y;
      c.kept_evals = ev;
      c.kept_start = k;
      c.kept_fault = __ldcg(w.fault + i);
      if (sf::lt(lowest, early)) break;
    }
  }
  return c;
}

}  // namespace photic
