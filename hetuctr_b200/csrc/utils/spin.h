// Waiting awake for a short time: waking a thread that has gone to sleep takes about ten microseconds, as long as the calls
// of a step follow each other.
#pragma once
#include <atomic>
#include <chrono>
#include <thread>

#if defined(__linux__)
#include <sched.h>
#include <sys/resource.h>
#endif

#include "utils/cpu_relax.h"

namespace hetuCTR {

// Processors the calling thread may run on, at least 1.
inline int processors() {
#if defined(__linux__)
  cpu_set_t set;
  if (sched_getaffinity(0, sizeof(set), &set) == 0) {
    const int n = CPU_COUNT(&set);
    if (n > 0) return n;
  }
#endif
  const unsigned n = std::thread::hardware_concurrency();
  return n > 0 ? (int)n : 1;
}

// How often the system has taken the processor from the calling thread for somebody else.
inline long pushed_aside() {
#if defined(__linux__)
  rusage u;
  if (getrusage(RUSAGE_THREAD, &u) == 0) return u.ru_nivcsw;
#endif
  return 0;
}

// Worker threads of the process's call queues.
inline std::atomic<int> &queue_workers() {
  static std::atomic<int> n{0};
  return n;
}

// Looks for `ready()` for up to `us` microseconds; true when it came.  A thread that waits awake must not keep from its work
// whoever it waits for:
//  * the `threads` that run together (waiting ones among them) have a processor each, or all of them sleep;
//  * a thread whose processor has been given to somebody else meanwhile - it looks every 16 waits - sleeps 64 times.
// Two and four ranks of 53,248 x 128 in one process and the thread that waits for them, us per pass, always awake (100 to
// 1000 us) -> so -> always asleep (an earlier build, 100 us slower elsewhere):
//   16 free processors       163 / 305 -> 166 / 305 -> 270 / 410       (3 threads / 5 threads)
//   as many as ranks         565 / 640 -> 210 / 341 -> 300 / 436
//   16, all computing       1600 / 2200 -> 480..760 / 730..1330 -> 670..830 / 1530..1790
template <class F>
inline bool spin_for(int us, int threads, F ready) {
  static thread_local int processors_here = 1, looks = 0, asleep = 0;
  static thread_local long pushed = 0;
  if (ready()) return true;
  if (asleep > 0) {
    asleep--;
    return false;
  }
  if (looks-- == 0) {  // (two system calls)
    looks = 15;
    processors_here = processors();
    const long seen = pushed_aside();
    if (seen != pushed) {
      pushed = seen;
      asleep = 63;
      looks = 0;
      return false;
    }
  }
  if (threads > processors_here) return false;
  const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(us);
  do {
    for (int i = 0; i < 32; i++) {
      cpu_relax();
      if (ready()) return true;
    }
  } while (std::chrono::steady_clock::now() < until);
  return false;
}

}  // namespace hetuCTR
