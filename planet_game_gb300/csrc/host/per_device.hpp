// What has to be found out or set once a device: a kernel's attributes
// (cudaFuncSetAttribute holds on the current device alone) and the limits that depend on it.
#pragma once

#include <map>
#include <mutex>
#include <utility>

namespace psgb {

// A value a device, made by `make()` when the device first asks. Safe with several threads;
// where `make` throws nothing is kept and the next call tries again.
template <typename V>
class PerDevice {
  public:
    template <typename Make>
    V of(int device, Make&& make) {
        std::lock_guard<std::mutex> lock(mu_);
        const auto found = made_.find(device);
        if (found != made_.end()) return found->second;
        return made_.emplace(device, std::forward<Make>(make)()).first->second;
    }

  private:
    std::mutex mu_;
    std::map<int, V> made_;
};

}  // namespace psgb
