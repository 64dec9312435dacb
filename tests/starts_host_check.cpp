// Host check of start_wanted (photic_starts.cuh): the lanes of a group, here
// threads, ask whether a depth start is still wanted while the word that says
// so falls between their loads.  All of them have to get the same answer:
// barriers and exchanges of the whole group follow it.  The shuffle is a
// rendezvous of the group's threads.
//
//   starts_host_check <rounds>
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>

#include <atomic>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

namespace {

constexpr int kLanes = 8;
thread_local int t_lane = 0;
pthread_barrier_t g_meet;
int g_slot[kLanes];
std::atomic<int> g_word{0}, g_loads{0};

}  // namespace

// Every load sees the word lower than the one before it did.
static inline int __ldcg(const int *) {
  g_loads++;
  return g_word.fetch_sub(1);
}
static inline double __ldcg(const double *p) { return *p; }
static inline int __shfl_sync(unsigned, int v, int from, int) {
  g_slot[t_lane] = v;
  pthread_barrier_wait(&g_meet);
  const int r = g_slot[from];
  pthread_barrier_wait(&g_meet);
  return r;
}
static inline void __threadfence() {}
static inline void __syncwarp(unsigned) { pthread_barrier_wait(&g_meet); }
static inline int atomicMin(int *p, int v) { return *p < v ? *p : (*p = v); }
static inline unsigned long long atomicOr(unsigned long long *p, unsigned long long v) {
  const unsigned long long o = *p;
  *p |= v;
  return o;
}
#include "photic_starts.cuh"

int main(int argc, char **argv) {
  const int rounds = argc > 1 ? atoi(argv[1]) : 100;
  pthread_barrier_init(&g_meet, nullptr, kLanes);
  int split = 0, wanted = 0;
  for (int n = 0; n < rounds; n++) {
    // the word passes the asked start within kLanes loads: from wanted to not
    const int start = 1 + n % 31;
    g_word = start + n % kLanes;
    g_loads = 0;
    int answer[kLanes];
    std::vector<std::thread> lanes;
    for (int l = 0; l < kLanes; l++)
      lanes.emplace_back([&, l] {
        t_lane = l;
        int32_t word = 0;
        answer[l] = photic::start_wanted(&word, start, 0xffu, kLanes, l);
      });
    for (std::thread &t : lanes) t.join();
    for (int l = 1; l < kLanes; l++) split += answer[l] != answer[0];
    wanted += answer[0];
    if (g_loads != 1) split++;
  }
  printf("%d rounds, %d wanted, %d answers differ\n", rounds, wanted, split);
  puts(split == 0 && wanted == rounds ? "OK" : "FAILED");
  return split != 0 || wanted != rounds;
}
