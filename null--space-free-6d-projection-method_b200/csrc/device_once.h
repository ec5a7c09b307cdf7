// Work that is done once per device, not once per process.
#pragma once
#include <atomic>

namespace fame {

// once(device, f): runs f until it has returned 0 for this device.  Two threads may both run it
// the first time, so f has to be repeatable.  Devices outside 0..63 run it every time.
class DeviceOnce {
  std::atomic<unsigned long long> done{0};

 public:
  template <class F> int operator()(int device, F f) {
    const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
    if (done.load(std::memory_order_relaxed) & bit) return 0;
    const int s = f();
    if (s == 0) done.fetch_or(bit, std::memory_order_relaxed);
    return s;
  }
};

}  // namespace fame
