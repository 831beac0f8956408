// Settings that belong to a device (a kernel's shared-memory limit): made on each
// device of the process that needs them, once.  Plain C++.
#pragma once

#include <mutex>

namespace lgb {

class OncePerDevice {
 public:
  // set() on the first call for `device`, and again after one that did not return `ok`
  template <typename Status, typename Set>
  Status run(int device, Status ok, Set set) {
    std::lock_guard<std::mutex> lock(mu_);
    const bool known = device >= 0 && device < MAX_DEVICES;
    if (known && done_[device]) return ok;
    const Status st = set();
    if (known && st == ok) done_[device] = true;
    return st;
  }

 private:
  static constexpr int MAX_DEVICES = 64;     // beyond: set on every call
  std::mutex mu_;
  bool done_[MAX_DEVICES] = {};
};

}  // namespace lgb
