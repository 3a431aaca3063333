// Which devices of a process have had a kernel's attributes set. They belong to
// one device each, so a flag for the process covers the first device only; and
// contexts on several host threads reach it at the same time.
#pragma once

#include <atomic>
#include <cstdint>

namespace bartels {

class DeviceOnce {
 public:
  bool pending(int device) const {
    return device < 0 || device >= 64 || !((done_.load(std::memory_order_acquire) >> device) & 1u);
  }
  // after the attributes are set; two threads may both have set them, to the same values
  void set(int device) {
    if (device >= 0 && device < 64) done_.fetch_or(uint64_t(1) << device, std::memory_order_release);
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace bartels
