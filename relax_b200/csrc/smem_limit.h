// The dynamic shared-memory limit of one kernel (cudaFuncAttributeMaxDynamicSharedMemorySize), as launches of any
// size from any thread need it.  The limit belongs to the kernel on one device and is shared by all threads of the process,
// so what it stands at is kept per device, and it is changed under a lock and only ever raised: a launch that was
// told that its size is allowed stays allowed, whatever other threads launch.
#pragma once
#include <stddef.h>

#include <atomic>
#include <mutex>

namespace b200 {

class SmemLimit {
 public:
  // Makes the limit at least `bytes` on device `dev`; `set(bytes)` changes it there and returns 0 where it could.
  template <class Set>
  int raise(int dev, size_t bytes, Set set) {
    const bool known = dev >= 0 && dev < kDevices;
    if (known && bytes <= limit_[dev].load(std::memory_order_acquire)) return 0;
    std::lock_guard<std::mutex> lock(mutex_);
    if (!known) return set(bytes);
    if (bytes <= limit_[dev].load(std::memory_order_relaxed)) return 0;
    const int rc = set(bytes);
    if (rc == 0) limit_[dev].store(bytes, std::memory_order_release);
    return rc;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<size_t> limit_[kDevices] = {};
  std::mutex mutex_;
};

}  // namespace b200
