#pragma once
#include <mutex>

namespace moe {

// One value per device, made on first use.
template <typename T>
class PerDevice {
 public:
  template <typename Make>
  const T* get(int device, Make make) {   // null: no such device
    if (device < 0 || device >= MAX) return nullptr;
    std::call_once(once_[device], [&] { value_[device] = make(device); });
    return value_ + device;
  }

 private:
  static constexpr int MAX = 64;
  std::once_flag once_[MAX];
  T value_[MAX];
};

}  // namespace moe
