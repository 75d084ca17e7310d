// One-time set-up of something that belongs to a device (a kernel's
// shared-memory limit, for instance): once per device, not per process, since
// contexts of one process may be on several.  Plain C++.
#pragma once

#include <cstdint>
#include <mutex>

namespace pyfof {

class PerDeviceOnce {
 public:
  static constexpr int kDevices = 64;
  // f() for `device` the first time it is asked for (concurrent callers wait);
  // its status every time.  -1: no such device number.
  template <class F>
  int32_t run(int device, F &&f) {
    if (device < 0 || device >= kDevices) return -1;
    std::call_once(once_[device], [&] { status_[device] = f(); });
    return status_[device];
  }

 private:
  std::once_flag once_[kDevices];
  int32_t status_[kDevices] = {};
};

}  // namespace pyfof
