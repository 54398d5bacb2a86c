// What a process sets once on each device that it uses: function attributes (they
// belong to the device that is current when they are set) and device properties.
#pragma once

#include <atomic>
#include <mutex>

namespace bem2d_gpu {

constexpr int kMaxDevices = 64;  // beyond: every time

// once(dev, f) calls f() if it has not yet returned for that device; callers of
// one device wait for it.
class PerDeviceOnce {
 public:
  template <typename F>
  void operator()(int dev, F f) {
    if (dev < 0 || dev >= kMaxDevices) {
      f();
      return;
    }
    if (done_[dev].load(std::memory_order_acquire)) return;
    std::lock_guard<std::mutex> lock(mu_);
    if (done_[dev].load(std::memory_order_relaxed)) return;
    f();
    done_[dev].store(true, std::memory_order_release);
  }

 private:
  std::mutex mu_;
  std::atomic<bool> done_[kMaxDevices] = {};
};

// A value for each device, `init` at first; devices beyond the last share one.
template <typename T>
class PerDevice {
 public:
  explicit PerDevice(T init) {
    for (auto& v : v_) v = init;
  }
  std::atomic<T>& operator[](int dev) {
    return v_[dev < 0 || dev >= kMaxDevices ? kMaxDevices : dev];
  }

 private:
  std::atomic<T> v_[kMaxDevices + 1];
};

}  // namespace bem2d_gpu
