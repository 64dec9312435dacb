// photic_workspace.h -- workspace that a call can do with less of.
//
// The fits keep a record per depth start so that the starts run beside each
// other, up to 1 GiB; without records a pixel's starts run one after another
// with the same result and need next to nothing.  Where the device has too
// little memory left, a call takes half as many records, and half again, down
// to none, instead of failing.
//
// The header compiles for the host alone (tests/workspace_host_check.cpp).
#pragma once
#include <stdint.h>

namespace photic {

enum class WsTry { kDone, kNoMemory, kFailed };

// attempt(n) for n, n / 2, ... and at last 0 (in the place of anything below
// `least`), until it does not end with kNoMemory; n is the one that did not.
template <class Attempt>
WsTry take_less(int64_t &n, int64_t least, Attempt &&attempt) {
  for (;;) {
    const WsTry t = attempt(n);
    if (t != WsTry::kNoMemory || n == 0) return t;
    n = n / 2 < least ? 0 : n / 2;
  }
}

}  // namespace photic
