// Short bounded polling before a thread goes to sleep.
//
// Requests on the device plane complete within microseconds; a condition variable costs several
// microseconds on either side of each hand-over.  Threads that expect such a completion poll for
// SpinMicros() first.  PSB200_SPIN_US sets the limit; a process that may use fewer than four
// CPUs does not poll (the polling thread would take the CPU of the one it waits for).
#ifndef PS_INTERNAL_SPIN_H_
#define PS_INTERNAL_SPIN_H_
#include <sched.h>

#include <chrono>
#include <cstdlib>
#include <mutex>

namespace ps {

inline int SpinMicros() {
  static const int us = [] {
    if (const char* e = getenv("PSB200_SPIN_US")) return atoi(e);
    cpu_set_t set;
    CPU_ZERO(&set);
    if (sched_getaffinity(0, sizeof(set), &set) == 0 && CPU_COUNT(&set) < 4) return 0;
    return 200;
  }();
  return us;
}

inline void CpuPause() {
#if defined(__x86_64__) || defined(__i386__)
  __builtin_ia32_pause();
#endif
}

// Takes a mutex that is held for less than a microsecond at a time: a thread that went to sleep
// on it would have to be woken by the holder, which costs either side more than the wait.
inline std::unique_lock<std::mutex> SpinLock(std::mutex& mu) {
  std::unique_lock<std::mutex> lk(mu, std::defer_lock);
  for (int i = 0; i < 64; ++i) {
    if (lk.try_lock()) return lk;
    CpuPause();
  }
  lk.lock();
  return lk;
}

// Polls `ready` until it holds or `until` has passed; returns whether it held.
template <typename F>
inline bool SpinUntil(std::chrono::steady_clock::time_point until, F&& ready) {
  for (;;) {
    for (int i = 0; i < 16; ++i) {
      if (ready()) return true;
      CpuPause();
    }
    if (std::chrono::steady_clock::now() >= until) return ready();
  }
}

}  // namespace ps
#endif  // PS_INTERNAL_SPIN_H_
