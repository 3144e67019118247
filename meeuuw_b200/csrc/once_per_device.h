// Work that every device of a process needs once before its first launch of something: a constant bank
// filled, a kernel's shared-memory limit raised.
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace mw {

class OncePerDevice {
 public:
  static constexpr int DEVICES = 64;

  // Calls work() for device `dev` (the caller's current one) unless it has succeeded there already; other
  // threads wait for it.  False when work() failed -- the next call tries again -- or there is no such device.
  template <typename F>
  bool run(int dev, const F& work) {
    if (dev < 0 || dev >= DEVICES) return false;
    const uint64_t bit = uint64_t(1) << dev;
    if (done_.load(std::memory_order_acquire) & bit) return true;
    std::lock_guard<std::mutex> lock(mutex_);
    if (done_.load(std::memory_order_relaxed) & bit) return true;
    if (!work()) return false;
    done_.fetch_or(bit, std::memory_order_release);
    return true;
  }

 private:
  std::atomic<uint64_t> done_{0};
  std::mutex mutex_;
};

}  // namespace mw
