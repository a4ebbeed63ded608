// per_device.h -- launch settings that hold for one device of the process: a
// kernel's shared-memory opt-in, the CTAs of it that fit an SM, a memory pool's
// configuration.
#pragma once

#include <mutex>

namespace vt {

// What `find` returns for a device, found on the first call for it (the calling
// thread's current device) and kept; safe with several threads.  A find that
// throws keeps nothing.
template <class T>
class PerDevice {
 public:
  template <class F>
  T get(int device, F&& find) {
    if (device < 0 || device >= kDevices) return find();
    std::call_once(once_[device], [&] { value_[device] = find(); });
    return value_[device];
  }

 private:
  static constexpr int kDevices = 64;
  std::once_flag once_[kDevices];
  T value_[kDevices] = {};
};

}  // namespace vt
