// Host check of take_less (photic_workspace.h) with allocators of every
// capacity: it asks for the wanted number first, never again for more than
// what has failed, takes half until something fits, comes down to none, and
// passes any other failure on at once.
#include <stdio.h>

#include <vector>

#include "photic_workspace.h"

using photic::WsTry;

int main() {
  int bad = 0;
  const int64_t least = 16, base = 8;  // bytes without a record; eight a record
  for (int64_t want : {0, 1, 15, 16, 100, 1000, 4097}) {
    for (int64_t room = 0; room < base + 8 * 5000; room += 7) {
      std::vector<int64_t> asked;
      int64_t n = want;
      const WsTry t = photic::take_less(n, least, [&](int64_t m) {
        asked.push_back(m);
        return base + 8 * m <= room ? WsTry::kDone : WsTry::kNoMemory;
      });
      bad += asked[0] != want;
      for (size_t i = 1; i < asked.size(); i++)
        bad += asked[i] != (asked[i - 1] / 2 < least ? 0 : asked[i - 1] / 2);
      bad += asked.back() != n;
      bad += (t == WsTry::kDone) != (room >= base);
      bad += t == WsTry::kDone && base + 8 * n > room;
      bad += t == WsTry::kNoMemory && n != 0;
    }
    int64_t n = want;
    int calls = 0;
    bad += photic::take_less(n, least, [&](int64_t) {
             calls++;
             return WsTry::kFailed;
           }) != WsTry::kFailed;
    bad += calls != 1 || n != want;
  }
  puts(bad ? "FAILED" : "OK");
  return bad != 0;
}
