// What has to be set up once on each device, such as a kernel's shared memory limit, which belongs to the function on the
// device that was current. Host code without CUDA, so that it can be checked by itself.
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>

namespace plume {

class OncePerDevice {
 public:
  // set_up() on the first call for `device`, 0 (success) from then on; a failure is returned and tried again at the next
  // call. Threads that call for a device meanwhile wait for it. Devices past the 64th are set up at every call.
  template <class SetUp>
  int run(int device, SetUp set_up) {
    const bool counted = device >= 0 && device < 64;
    const uint64_t bit = counted ? uint64_t(1) << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    std::lock_guard<std::mutex> lock(mutex_);
    if (done_.load(std::memory_order_relaxed) & bit) return 0;
    const int status = set_up();
    if (status == 0) done_.fetch_or(bit, std::memory_order_release);
    return status;
  }

 private:
  std::mutex mutex_;
  std::atomic<uint64_t> done_{0};
};

}  // namespace plume
