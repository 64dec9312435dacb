// photic_ncrange.h -- when one pass over a grid gives compress_2d's maximum.
//
// compress_2d (model/nc.c:284-297) compares a cell with the maximum only if it
// does not lower the running minimum, so its maximum leaves out the grid's
// leading strictly decreasing run of compared cells (neither missing nor NaN)
// and nothing else that matters (nc_range_kernel, photic_ncgrid.cu).  The pass
// follows that run through a window at the grid's beginning.  Where it does
// not end there, mostly because the scene has a border without data and the
// run has not begun, the cells behind the window still tell.
//
// The header compiles for the host too (tests/ncrange_host_check.cpp).
#pragma once
#include <float.h>

#if defined(__CUDACC__)
#define PHOTIC_NR_HD __host__ __device__ inline
#else
#define PHOTIC_NR_HD inline
#endif

namespace photic {

enum : unsigned {
  kRangeKnown = 0,  // the pass's maximum is compress_2d's
  kRangeAll = 1,    // every cell has to be compared in order
  kRangeFirst = 2,  // the first compared cell decides (range_after_first)
};

// open: the run did not end in the window and the grid goes on behind it;
// run: the running minimum at the window's end (FLT_MAX: the window has no
// compared cell that lowers it); lo: the grid's minimum; hi: the maximum of
// FLT_MIN and, where open, the cells behind the window.
PHOTIC_NR_HD unsigned range_after_window(bool open, float run, float lo, float hi) {
  // what goes on with the run lies below its minimum so far, so a cell that
  // is not has been compared with the maximum
  if (!open || hi >= run) return kRangeKnown;
  if (run < FLT_MAX) return kRangeAll;
  return lo < FLT_MAX ? kRangeFirst : kRangeKnown;  // (or no cell at all is compared)
}

// The run begins at the first compared cell and falls from there.
PHOTIC_NR_HD unsigned range_after_first(float first, float hi) {
  return hi > first ? kRangeKnown : kRangeAll;
}

}  // namespace photic
