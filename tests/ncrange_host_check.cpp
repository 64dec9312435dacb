// Host check of photic_ncrange.h: the pass of nc_range_kernel and
// nc_first_kernel restated in order over small random grids, with a window of
// eight cells, and what the header says of its maximum, against compress_2d's
// loop (model/nc.c:284-297) as it stands there.  Where the header takes the
// pass's maximum it has to be that loop's; and it has to take it for every grid
// with a border without data whose first cell behind it is not the largest.
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <vector>

#include "photic_ncrange.h"

namespace {
uint64_t g_state = 7;
uint32_t next(uint32_t n) {
  g_state += 0x9e3779b97f4a7c15ULL;
  uint64_t z = g_state;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return (uint32_t)((z ^ (z >> 31)) % n);
}
}  // namespace

int main() {
  constexpr int kLead = 8;
  const float sp = -9.0f;
  const float values[] = {sp,       NAN,  -3.0f, -1.0f, 0.0f,     1.0f,      2.0f,
                          FLT_MIN,  5.0f, 8.0f,  1e30f, FLT_MAX,  INFINITY,  -INFINITY,
                          -FLT_MAX, 3.0f, 4.0f,  6.0f,  FLT_MIN / 2, 7.0f};
  const uint32_t count = sizeof values / sizeof *values;
  long bad = 0, known = 0, all = 0, first = 0, borders = 0;
  for (int trial = 0; trial < 2000000; trial++) {
    const int n = 1 + (int)next(24);
    std::vector<float> g(n);
    const uint32_t kind = next(4);
    const int border = kind & 1 ? (int)next(n + 1) : 0;
    const int run = kind & 2 ? border + (int)next(n + 1) : 0;
    for (int i = 0; i < n; i++)
      g[i] = i < border ? (next(9) ? sp : NAN) : i < run ? (float)(40 - i) : values[next(count)];
    // compress_2d
    float grmin = FLT_MAX, grmax = FLT_MIN;
    for (float v : g) {
      if (v == sp) continue;
      if (v < grmin) grmin = v;
      else if (v > grmax) grmax = v;
    }
    // the pass
    const int head = n < kLead ? n : kLead;
    int lead = -1;
    float low = FLT_MAX, lo = FLT_MAX, hi = FLT_MIN;
    for (int i = 0; i < head && lead < 0; i++) {
      if (g[i] == sp || g[i] != g[i]) continue;
      if (g[i] < low) low = g[i];
      else lead = i;
    }
    const bool open = lead < 0 && n > kLead;
    if (lead < 0) lead = head;
    for (int i = 0; i < n; i++) {
      if (g[i] == sp) continue;
      if (g[i] < lo) lo = g[i];
      if (i >= lead && g[i] > hi) hi = g[i];
    }
    unsigned r = photic::range_after_window(open, low, lo, hi);
    float behind = NAN;  // the first compared cell
    for (int i = 0; i < n && behind != behind; i++)
      if (g[i] != sp) behind = g[i];
    if (r == photic::kRangeFirst) {
      first++;
      if (behind != behind) bad++;  // it is asked for where there is one
      r = photic::range_after_first(behind, hi);
    }
    if (r == photic::kRangeKnown) {
      known++;
      if (lo != grmin || hi != grmax) {
        if (bad++ < 5) printf("n %d: %g .. %g, want %g .. %g\n", n, lo, hi, grmin, grmax);
      }
    } else {
      all++;
      if (border >= kLead) {
        float most = -INFINITY;
        for (int i = 0; i < n; i++)
          if (g[i] != sp && g[i] > most) most = g[i];
        if (behind < most && most > FLT_MIN) bad++;
      }
    }
    borders += border >= kLead && n > kLead;
  }
  printf("%ld known, %ld of them from the first cell, %ld left, %ld borders, %ld wrong\n", known,
         first, all, borders, bad);
  puts(bad == 0 && first > 1000 && all > 1000 ? "OK" : "FAILED");
  return bad != 0;
}
