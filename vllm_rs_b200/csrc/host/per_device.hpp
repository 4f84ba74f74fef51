// What a process sets once per CUDA device: kernel attributes belong to the device that was current when they were set.
#pragma once
#include <atomic>
#include <cstdint>

namespace b200 {

// First call per device runs `set` and, if that succeeds, no later call does; a failure is returned and tried again next time.
// Threads may meet in it: setting the same attribute twice does no harm.
class OncePerDevice {
  std::atomic<uint64_t> done_{0};

 public:
  template <typename F>
  auto operator()(int device, F set) -> decltype(set()) {
    const bool counted = device >= 0 && device < 64;
    const uint64_t bit = counted ? uint64_t{1} << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return decltype(set()){};
    const auto error = set();
    if (error == decltype(set()){}) done_.fetch_or(bit, std::memory_order_release);
    return error;
  }
};

}  // namespace b200
