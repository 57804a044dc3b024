// A number that belongs to a device: asked for once per device, whichever threads and devices come first.  Plain C++.
#pragma once

#include <mutex>

namespace gca {

class PerDevice {
 public:
  static constexpr int MAX_DEVICES = 64;
  // `ask(&value)` says whether it found out.  A failed attempt is not kept: the next call asks again.
  template <class F>
  bool get(int dev, int* value, F&& ask) {
    if (dev < 0 || dev >= MAX_DEVICES) return ask(value);
    std::lock_guard<std::mutex> lock(mu_);
    if (!known_[dev]) {
      int v = 0;
      if (!ask(&v)) return false;
      value_[dev] = v;
      known_[dev] = true;
    }
    *value = value_[dev];
    return true;
  }

 private:
  std::mutex mu_;
  int value_[MAX_DEVICES] = {};
  bool known_[MAX_DEVICES] = {};
};

}  // namespace gca
