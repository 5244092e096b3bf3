// A value made once per device, at its first use there (thread-safe): kernel attributes hold for the
// device that was current when they were set, and occupancies and SM counts for the one that was asked.
#pragma once

#include <array>
#include <mutex>

#include "host.hpp"

namespace fx {

constexpr int kMaxDevices = 64;

template <class T>
class PerDevice {
 public:
  // make(): the value for `device`, called at the first get for it (again after a call that threw)
  template <class Make>
  T get(int device, Make&& make) {
    if (device < 0 || device >= kMaxDevices) throw Error(FX_E_UNSUPPORTED, "device index past the 64 this build holds");
    std::call_once(once_[device], [&] { value_[device] = make(); });
    return value_[device];
  }

 private:
  std::array<std::once_flag, kMaxDevices> once_;
  std::array<T, kMaxDevices> value_{};
};

}  // namespace fx
