// What has been done once per device: a kernel's attributes hold for the device that is
// current when they are set, and engines on several devices may launch from several threads.
#pragma once

#include <atomic>
#include <cstdint>

namespace fhe_b200 {

class DeviceOnce {
 public:
  bool done(int device) const {
    return device >= 0 && device < 64 && ((devices_.load(std::memory_order_acquire) >> device) & 1) != 0;
  }
  // Devices from 64 on are never done: their attributes are set again by every call.
  void set_done(int device) {
    if (device >= 0 && device < 64) devices_.fetch_or(uint64_t(1) << device, std::memory_order_release);
  }

 private:
  std::atomic<uint64_t> devices_{0};
};

}  // namespace fhe_b200
