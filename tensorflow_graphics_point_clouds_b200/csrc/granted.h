// The most a resource has been raised to so far, asked for once per larger size.
// Host alone, without CUDA headers.
#pragma once

#include <atomic>
#include <mutex>

namespace tfgpc {

class Granted {
 public:
  // 0 once at least `size` is granted, else what ask(size) returned.  One thread asks at a time
  // and none for less than another has been given: asked for a smaller size in between, the
  // driver would hold that one and every later call rely on the larger.
  template <typename Ask>
  int reach(int size, Ask ask) {
    if (size <= most_.load(std::memory_order_acquire)) return 0;
    std::lock_guard<std::mutex> hold(lock_);
    if (size <= most_.load(std::memory_order_relaxed)) return 0;
    const int e = ask(size);
    if (e == 0) most_.store(size, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<int> most_{0};
  std::mutex lock_;
};

}  // namespace tfgpc
