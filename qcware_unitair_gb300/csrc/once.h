// Work that is to be done once on each device.
#pragma once

#include <stdint.h>

#include <atomic>

namespace gbsv {

// Runs f() for a device until it has returned 0 there, and returns what it
// returned, 0 afterwards.  Threads may run it at the same time; none goes on
// before it is done on its device.
struct OncePerDevice {
  std::atomic<uint64_t> done{0};
  template <typename F>
  int operator()(int device, F f) {
    if (device >= 0 && device < 64 &&
        ((done.load(std::memory_order_acquire) >> device) & 1))
      return 0;
    const int rc = f();
    if (rc == 0 && device >= 0 && device < 64)
      done.fetch_or(uint64_t(1) << device, std::memory_order_release);
    return rc;
  }
};

}  // namespace gbsv
