// How much dynamic shared memory one kernel may be launched with, per device.
#pragma once

#include <atomic>
#include <cstddef>
#include <mutex>

namespace tpb {
namespace kernels {

// A limit that is only ever raised. Several threads launch the same kernel with different needs, and the
// driver keeps the LAST value it was given, so setting a limit and remembering it must be one step: a thread
// that sets a smaller one between the two would leave the kernel with less than what is remembered.
class SmemLimit {
 public:
  // On return a launch with `bytes` on `device` is allowed; `set(bytes)` is called if it was not. What
  // `set` throws goes to the caller and nothing is remembered.
  template <typename F>
  void raise(int device, size_t bytes, F&& set) {
    if (device < 0 || device >= kDevices) return;
    std::atomic<size_t>& allowed = allowed_[device];
    if (allowed.load(std::memory_order_acquire) >= bytes) return;
    std::unique_lock<std::mutex> lock(mutex_);
    if (allowed.load(std::memory_order_relaxed) >= bytes) return;
    set(bytes);
    allowed.store(bytes, std::memory_order_release);
  }

 private:
  static constexpr int kDevices = 64;
  std::mutex mutex_;
  std::atomic<size_t> allowed_[kDevices] = {};
};

}  // namespace kernels
}  // namespace tpb
