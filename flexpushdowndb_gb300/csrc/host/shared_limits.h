// The dynamic shared-memory limits that kernels have been given.
//
// A kernel's limit belongs to the kernel on a device: it is one value for all
// threads and stays between a call's setting it and its launch. So it is only
// ever raised, under a lock: a call that needs less leaves it alone, and a
// launch never finds it below what its own call asked for.
#pragma once

#include <map>
#include <mutex>
#include <utility>

namespace gfpdb {

class SharedLimits {
 public:
  // Calls set(bytes) when the kernel's limit on the device is below `bytes`;
  // one that throws leaves the limit as it was.
  template <class Set>
  void raise(int device, const void* kernel, int bytes, Set&& set) {
    std::lock_guard<std::mutex> lk(mu_);
    int& limit = limits_[{device, kernel}];
    if (bytes <= limit) return;
    set(bytes);
    limit = bytes;
  }

 private:
  std::mutex mu_;
  std::map<std::pair<int, const void*>, int> limits_;
};

}  // namespace gfpdb
