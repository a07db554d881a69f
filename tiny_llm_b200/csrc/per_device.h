// What has to be set up once per device of the process, for instance the limit of a kernel's dynamic shared memory:
// cudaFuncSetAttribute holds for the device that is current.  Plain C++, no CUDA.
#pragma once
#include <atomic>
#include <mutex>

namespace tllm {

// The largest value that has been set on each device.
class PerDeviceLimit {
 public:
  static constexpr int DEVICES = 64;
  // Calls set(), which returns 0 or an error code, unless `value` or more has been set on `device`.  A set() that fails is
  // not noted; ordinals that have no place here are set at every call.
  template <typename Set>
  int raise(int device, long long value, Set set) {
    if (device < 0 || device >= DEVICES) return set();
    if (limit_[device].load(std::memory_order_acquire) >= value) return 0;
    std::lock_guard<std::mutex> hold(setup_);
    if (limit_[device].load(std::memory_order_relaxed) >= value) return 0;
    const int e = set();
    if (e == 0) limit_[device].store(value, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<long long> limit_[DEVICES] = {};
  std::mutex setup_;
};

}  // namespace tllm
