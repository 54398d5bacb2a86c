// A few host threads that share a loop's iterations, for the length of one
// call (the numerical range analyses hundreds of small tridiagonals between
// two GPU steps).
#pragma once

#include <atomic>
#include <condition_variable>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace bem2d_gpu {

class HostPool {
 public:
  // `threads` workers beside the caller; fewer if the system refuses some.
  explicit HostPool(int threads) {
    for (int i = 0; i < threads; ++i) {
      try {
        workers_.emplace_back([this] { work(); });
      } catch (...) {
        break;
      }
    }
  }
  ~HostPool() {
    {
      std::lock_guard<std::mutex> lock(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : workers_) t.join();
  }
  HostPool(const HostPool&) = delete;
  HostPool& operator=(const HostPool&) = delete;

  // fn(0) .. fn(n - 1) in any order on any of the threads; false if one threw.
  bool run(int n, const std::function<void(int)>& fn) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      fn_ = &fn;
      n_ = n;
      next_ = 0;
      failed_ = false;
      busy_ = (int)workers_.size();
      ++round_;
    }
    wake_.notify_all();
    drain();
    std::unique_lock<std::mutex> lock(mu_);
    done_.wait(lock, [this] { return busy_ == 0; });
    return !failed_;
  }

 private:
  void drain() {
    try {
      for (int i; (i = next_.fetch_add(1)) < n_;) (*fn_)(i);
    } catch (...) {
      failed_ = true;
      next_ = n_;
    }
  }
  void work() {
    long long seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lock(mu_);
        wake_.wait(lock, [&] { return stop_ || round_ != seen; });
        if (stop_) return;
        seen = round_;
      }
      drain();
      std::lock_guard<std::mutex> lock(mu_);
      if (--busy_ == 0) done_.notify_one();
    }
  }

  std::vector<std::thread> workers_;
  std::mutex mu_;
  std::condition_variable wake_, done_;
  const std::function<void(int)>* fn_ = nullptr;
  std::atomic<int> next_{0};
  std::atomic<bool> failed_{false};
  int n_ = 0, busy_ = 0;
  long long round_ = 0;
  bool stop_ = false;
};

}  // namespace bem2d_gpu
