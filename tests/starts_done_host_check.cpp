// Host check of start_done (photic_starts.cuh): the lanes of a group, here
// threads, publish a start and are told whether theirs is the one that compares
// the pixel's records.  All lanes get one answer; one group of the pixel's gets
// it; and every lane meets its fence and a barrier before the first lane
// publishes, and a barrier after the answer is handed on, before it reads.
//
//   starts_done_host_check <pixels>
#include <math.h>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>

#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

namespace {
constexpr int kLanes = 8;
struct Group {
  pthread_barrier_t meet;
  int slot;
};
thread_local int t_lane = 0;
thread_local Group *t_group = nullptr;
thread_local std::string t_events;
std::mutex g_memory;
}  // namespace

static inline int __ldcg(const int *p) {
  std::lock_guard<std::mutex> l(g_memory);
  return *p;
}
static inline double __ldcg(const double *p) { return *p; }
static inline int __shfl_sync(unsigned, int v, int from, int) {
  if (t_lane == from) t_group->slot = v;
  pthread_barrier_wait(&t_group->meet);
  const int r = t_group->slot;
  pthread_barrier_wait(&t_group->meet);
  t_events += 'x';
  return r;
}
static inline void __syncwarp(unsigned) {
  pthread_barrier_wait(&t_group->meet);
  t_events += 'b';
}
static inline void __threadfence() { t_events += 'f'; }
static inline int atomicMin(int *p, int v) {
  std::lock_guard<std::mutex> l(g_memory);
  const int o = *p;
  if (v < o) *p = v;
  t_events += 'p';
  return o;
}
static inline unsigned long long atomicOr(unsigned long long *p, unsigned long long v) {
  std::lock_guard<std::mutex> l(g_memory);
  const unsigned long long o = *p;
  *p |= v;
  t_events += 'p';
  return o;
}
#include "photic_starts.cuh"

int main(int argc, char **argv) {
  const int pixels = argc > 1 ? atoi(argv[1]) : 50;
  constexpr int kStarts = 4;
  long bad = 0, chosen = 0;
  for (int p = 0; p < pixels; p++) {
    unsigned long long done = 0;
    int exit_k = 0x7f7f7f7f;
    photic::StartWork w = {};
    w.done = &done;
    w.exit_k = &exit_k;
    // every seventh pixel: a start meets the exit
    const int exits = p % 7 == 0 ? p % kStarts : -1;
    Group groups[kStarts];
    int answer[kStarts][kLanes];
    std::string events[kStarts][kLanes];
    std::vector<std::thread> threads;
    for (int k = 0; k < kStarts; k++) pthread_barrier_init(&groups[k].meet, nullptr, kLanes);
    for (int k = 0; k < kStarts; k++)
      for (int l = 0; l < kLanes; l++)
        threads.emplace_back([&, k, l] {
          t_lane = l;
          t_group = &groups[k];
          t_events.clear();
          answer[k][l] = photic::start_done(w, 0, k, kStarts, k == exits ? 1.0 : 9.0, 2.0, 0xffu,
                                            kLanes, l);
          events[k][l] = t_events;
        });
    for (std::thread &t : threads) t.join();
    int took = 0;
    for (int k = 0; k < kStarts; k++) {
      took += answer[k][0];
      for (int l = 0; l < kLanes; l++) {
        const std::string &e = events[k][l];
        bad += answer[k][l] != answer[k][0];
        const size_t first = e.find('b'), published = e.find('p'), told = e.find('x');
        bad += e.find('f') > first;                                  // fence, then barrier,
        bad += published != std::string::npos && published < first;  // then it is published;
        bad += told == std::string::npos || e.find('b', told) == std::string::npos;
      }
    }
    bad += took != 1;
    chosen += took;
  }
  printf("%d pixels, %ld chosen, %ld wrong\n", pixels, chosen, bad);
  puts(bad == 0 ? "OK" : "FAILED");
  return bad != 0;
}
