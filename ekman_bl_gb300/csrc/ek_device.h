// Settings that CUDA keeps per device (a kernel's shared-memory limit, the SM
// count) made once for each device a process uses.
#pragma once

#include <mutex>

namespace ek {

class OncePerDevice {
 public:
  // f() for the first call with this device; a call that throws is made again.
  // Devices beyond the table run f each time.
  template <typename F>
  void operator()(int device, F &&f) {
    if (device < 0 || device >= kDevices) f();
    else std::call_once(flag_[device], f);
  }

 private:
  static constexpr int kDevices = 128;
  std::once_flag flag_[kDevices];
};

}  // namespace ek
