// What a kernel may have of shared memory on each device, beyond the 48 KiB that every launch may ask for.
#pragma once
#include <atomic>
#include <cstddef>
#include <mutex>

// The attribute is per device and sticky, and setting it lower takes back what was granted.  So it is asked for once per device and
// again only for more, by one thread at a time: two threads that set it for tiles of different sizes could otherwise leave the lower
// value in force with the higher one noted, and every later launch of the larger tile would be refused.
class SmemGrant {
 public:
  // `set(bytes)` asks the driver; returns 0 or its error.
  template <typename SET>
  int ask(int dev, size_t bytes, SET&& set) {
    std::atomic<size_t>* slot = dev >= 0 && dev < kDevices ? &granted_[dev] : nullptr;
    if (slot != nullptr && slot->load(std::memory_order_acquire) >= bytes) return 0;
    std::lock_guard<std::mutex> g(mu_);
    if (slot != nullptr && slot->load(std::memory_order_relaxed) >= bytes) return 0;
    const int e = set(bytes);
    if (e == 0 && slot != nullptr) slot->store(bytes, std::memory_order_release);
    return e;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<size_t> granted_[kDevices]{};
  std::mutex mu_;
};
