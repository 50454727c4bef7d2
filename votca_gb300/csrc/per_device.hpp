// Work done once per device of the process (a kernel's attributes belong to a device).
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace vgb {

class PerDevice {
 public:
  // f() on the first call with this device, and on every call for devices beyond the 64 that are counted;
  // again on the next call when f throws.
  template <class F>
  void run(int device, F &&f) {
    const uint64_t bit = device >= 0 && device < 64 ? 1ull << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return;
    std::lock_guard<std::mutex> lk(mu_);
    if (done_.load(std::memory_order_relaxed) & bit) return;
    f();
    done_.fetch_or(bit, std::memory_order_release);
  }

 private:
  std::mutex mu_;
  std::atomic<uint64_t> done_{0};
};

}  // namespace vgb
