// Setup that each device of the process needs once (kernel attributes).
#pragma once

#include <mutex>

namespace gi {

class OncePerDevice {
 public:
  // fn() (0: done) the first time for this device, and again after a failure.
  template <class F>
  auto run(int device, F&& fn) -> decltype(fn()) {
    std::lock_guard<std::mutex> lk(mu_);
    if (device >= 0 && device < kDevices && done_[device]) return decltype(fn())(0);
    const auto status = fn();
    if (device >= 0 && device < kDevices) done_[device] = (int)status == 0;
    return status;
  }

 private:
  static constexpr int kDevices = 64;  // more are set up on every call
  std::mutex mu_;
  bool done_[kDevices] = {};
};

}  // namespace gi
