// per_device.h -- values found out once for each device of a process (what a
// kernel's attributes were set to, how many of its CTAs fit an SM): a function
// attribute holds for the device that was current when it was set, and other
// devices may differ.  Plain code without CUDA types.
#pragma once

#include <mutex>

namespace grus {

template <class T>
class PerDevice {
 public:
  // The value of device `dev`, from find(value), which returns 0 where it worked.
  // A failure is returned and not kept.
  template <class Find>
  int get(int dev, T *out, Find find) {
    if (dev < 0 || dev >= kMax) return find(*out);
    std::lock_guard<std::mutex> lk(mu_);
    if (!known_[dev]) {
      T v{};
      const int rc = find(v);
      if (rc) return rc;
      value_[dev] = v;
      known_[dev] = true;
    }
    *out = value_[dev];
    return 0;
  }

 private:
  static constexpr int kMax = 64;
  std::mutex mu_;
  T value_[kMax] = {};
  bool known_[kMax] = {};
};

}  // namespace grus
