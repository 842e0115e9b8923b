// Work that each device needs once: function attributes belong to a device's context. Handles on one device may be used
// from several threads, each under its own handle's lock only, so the marks are atomic; threads that come together may do
// the work twice, which is harmless for what it is used for.
#pragma once
#include <atomic>
#include <stdint.h>

namespace cla {

struct OncePerDevice {
  static constexpr int DEVICES = 64;  // further devices do the work each time
  std::atomic<bool> done[DEVICES] = {};
  // work: returns a negative status when it failed (it is then tried again by the next caller)
  template <class F>
  int64_t operator()(int device, F&& work) {
    const bool marked = device >= 0 && device < DEVICES;
    if (marked && done[device].load(std::memory_order_acquire)) return 0;
    const int64_t rc = work();
    if (rc >= 0 && marked) done[device].store(true, std::memory_order_release);
    return rc;
  }
};

}  // namespace cla
