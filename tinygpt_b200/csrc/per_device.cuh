// per_device.cuh — what is set once for each device and not once for a process: a kernel's attributes hold for the device that is current when they are set.
// Plain C++, for the host alone.
#pragma once

#include <atomic>

namespace b200 {

// Error: a status whose value-initialised form says that all is well
template <typename Error, int kDevices = 64>
class OncePerDevice {
 public:
  // calls `set` until it has succeeded on this device (threads that come at once may all call it), every time on one past the table
  template <typename F>
  Error operator()(int device, F set) {
    const bool listed = device >= 0 && device < kDevices;
    if (listed && done_[device].load(std::memory_order_acquire)) return Error{};
    const Error e = set();
    if (listed && e == Error{}) done_[device].store(true, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<bool> done_[kDevices] = {};
};

}  // namespace b200
