// Facts about a kernel that hold per device (its dynamic shared memory limit, how many of its CTAs
// are resident), found once on each. A process may drive contexts on several devices, from several
// threads.
#pragma once

#include <atomic>

namespace lee {

class PerDevice {
 public:
  // The value kept for the device, or make()'s, kept when it is positive (a failure is tried again).
  // Two threads may both make it; they make the same.
  template <typename F>
  int get(int device, F&& make) {
    if (device < 0 || device >= kDevices) return make();
    int v = v_[device].load(std::memory_order_acquire);
    if (v <= 0) {
      v = make();
      if (v > 0) v_[device].store(v, std::memory_order_release);
    }
    return v;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<int> v_[kDevices] = {};
};

}  // namespace lee
