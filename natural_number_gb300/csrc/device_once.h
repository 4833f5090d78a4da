// device_once.h — work that every device of the process needs once, such as a
// kernel's attributes (which belong to the device that was current when they
// were set).  Only success is remembered: a failure is tried again by the next
// call.  No CUDA here, so that the CPU tests run the same code.
#pragma once

#include <atomic>
#include <cstdint>

namespace nn {

class DeviceOnce {
  static constexpr int kDevices = 64;  // beyond: set again each time
  std::atomic<uint64_t> done_{0};

 public:
  // `ok`, or what set() returned where this is not it.  Two threads may both
  // call set() the first time.
  template <class Status, class Set>
  Status operator()(int device, Status ok, const Set& set) {
    const uint64_t bit = device >= 0 && device < kDevices ? 1ull << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return ok;
    const Status s = set();
    if (s == ok) done_.fetch_or(bit, std::memory_order_release);
    return s;
  }
};

}  // namespace nn
