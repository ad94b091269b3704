// The largest dynamic shared memory a kernel has been allowed, for every device of the process: the limit belongs to the device, and
// several threads may be the first to launch a kernel.  It is only ever raised, under a lock, so that no thread takes back what
// another has set between its own request and its launch.
#pragma once

#include <cstdint>
#include <mutex>

namespace cmld {

class SmemLimit {
 public:
  // `set(bytes)` sets the limit of the current device, `dev`, and returns 0 when that worked.
  template <typename Set>
  int32_t raise(int dev, int bytes, Set &&set) {
    std::lock_guard<std::mutex> hold(lock_);
    const bool known = dev >= 0 && dev < kDevices;
    if (known && bytes <= allowed_[dev]) return 0;
    const int32_t rc = set(bytes);
    if (rc == 0 && known) allowed_[dev] = bytes;
    return rc;
  }

 private:
  static constexpr int kDevices = 64;  // (beyond: set every time)
  std::mutex lock_;
  int allowed_[kDevices] = {};
};

}  // namespace cmld
