// Work that each device needs once per process (a kernel's shared-memory
// limit, which CUDA keeps per device).
#pragma once

#include <cstdint>
#include <mutex>

namespace mts {

class DeviceOnce {
 public:
  // Runs f on this device unless it has succeeded there before; a second
  // caller waits for the first.  Returns f's error (0: none), which leaves
  // the work to be done by the next caller.
  template <class F>
  int run(int device, F f) {
    std::lock_guard<std::mutex> hold(lock_);
    const bool known = device >= 0 && device < 64;
    if (known && ((done_ >> device) & 1)) return 0;
    const int e = (int)f();
    if (e == 0 && known) done_ |= uint64_t(1) << device;
    return e;
  }

 private:
  std::mutex lock_;
  uint64_t done_ = 0;
};

}  // namespace mts
