// What has been set once per (device, kernel) pair: function attributes belong to
// a device, so a process that works on several of them sets each on every one.
#pragma once
#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace impes {

class DeviceLimits {
 public:
  // Calls set(value) unless the pair already holds at least `value`, and keeps the
  // value when set returned (an exception leaves the old one).  Host threads that
  // launch the same kernel with different sizes do not undo each other's setting.
  template <typename F>
  void raise(int device, const void* kernel, size_t value, F&& set) {
    std::lock_guard<std::mutex> lock(mu_);
    size_t& now = held_[{device, kernel}];
    if (value <= now) return;
    set(value);
    now = value;
  }

 private:
  std::mutex mu_;
  std::map<std::pair<int, const void*>, size_t> held_;
};

}  // namespace impes
