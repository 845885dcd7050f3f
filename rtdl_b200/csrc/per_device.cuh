// per_device.cuh -- handles made once per device (host code, no CUDA calls).
#pragma once

#include <map>
#include <utility>

namespace rtdl_b200 {

// Streams and events belong to the device that was current when they were made
// and serve on no other, so what a thread keeps of them is kept per device.
template <typename T>
class PerDevice {
 public:
  // Handle `which` of `device`; make() gives it on first use (nothing is kept
  // when it throws).
  template <typename Make>
  T get(int device, int which, Make&& make) {
    const std::pair<int, int> key(device, which);
    const auto it = made_.find(key);
    if (it != made_.end()) return it->second;
    const T made = make();
    made_.emplace(key, made);
    return made;
  }

 private:
  std::map<std::pair<int, int>, T> made_;
};

}  // namespace rtdl_b200
