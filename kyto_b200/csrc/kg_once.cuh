// Settings that belong to a pair of a kernel and a device. Plain C++: host code too.
#pragma once

#include <mutex>
#include <set>
#include <utility>

namespace kg {

// Runs a setting the first time a (key, device) pair comes by, from any thread; one that throws
// is tried again the next time. (A once_flag a kernel sets it on the process's first device only.)
class OncePerDevice {
 public:
  template <class Set>
  void operator()(const void* key, int device, Set&& set) {
    std::lock_guard<std::mutex> lock(mu_);
    const auto pair = std::make_pair(key, device);
    if (done_.count(pair)) return;
    set();
    done_.insert(pair);
  }

 private:
  std::mutex mu_;
  std::set<std::pair<const void*, int>> done_;
};

}  // namespace kg
