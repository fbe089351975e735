// cj_once.h -- set-up that belongs to a device and is made once for each.
#pragma once
#include <stdint.h>

#include <atomic>

// Runs f() for `device` until it has succeeded there (0): a kernel's function
// attributes, for instance, which are kept per device.  From any thread; two that
// come first at the same time may both run it.
struct CJOncePerDevice {
  std::atomic<uint64_t> done{0};  // bit per device; devices past 63 run it each time
  template <class F>
  auto run(int device, F f) -> decltype(f()) {
    const uint64_t bit = device >= 0 && device < 64 ? 1ull << device : 0;
    if (done.load(std::memory_order_acquire) & bit) return decltype(f())(0);
    const auto e = f();
    if (e == decltype(f())(0)) done.fetch_or(bit, std::memory_order_release);
    return e;
  }
};
