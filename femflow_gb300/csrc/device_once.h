// Set-up that belongs to a device (a kernel's attributes are those of the device that is current when they
// are set), done once per device and key by whichever thread comes first.
#pragma once

#include <mutex>
#include <set>
#include <utility>

namespace ffmpm {

class DeviceOnce {
 public:
  // True when set() has succeeded for (device, key), now or before.  One that failed is tried again.
  template <typename F>
  bool run(int device, const void* key, F&& set) {
    std::lock_guard<std::mutex> lock(mu_);
    const auto at = std::make_pair(device, key);
    if (done_.count(at)) return true;
    if (!set()) return false;
    done_.insert(at);
    return true;
  }

 private:
  std::mutex mu_;
  std::set<std::pair<int, const void*>> done_;
};

}  // namespace ffmpm
