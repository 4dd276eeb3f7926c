// Set-up that belongs to a device (function attributes, device properties),
// done on the first use of each device by a process.
#pragma once

#include <mutex>

namespace dense_b200 {

class PerDevice {
 public:
  // Runs set_up() (0: success) unless it succeeded on this device before;
  // its result.  Devices past the table run it every time.
  template <typename F>
  auto once(int device, F&& set_up) -> decltype(set_up()) {
    using R = decltype(set_up());
    if (device < 0 || device >= kDevices) return set_up();
    std::lock_guard<std::mutex> lock(mu_);
    if (done_[device]) return R(0);
    const R r = set_up();
    done_[device] = r == R(0);
    return r;
  }

 private:
  static constexpr int kDevices = 64;
  std::mutex mu_;
  bool done_[kDevices] = {};
};

}  // namespace dense_b200
