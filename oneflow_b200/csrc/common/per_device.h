// Setting something once for every device of the process. What cudaFuncSetAttribute sets (a kernel's limit of dynamic shared
// memory) belongs to the device that is current at the time: a flag per process leaves every other device without it.
#pragma once
#include <atomic>
#include <cstdint>

namespace ofb {

class OncePerDevice {
 public:
  // Calls `set` unless it has succeeded (returned 0) for this device before. Threads that come at the same time may both call it;
  // devices beyond the 64 that are remembered call it every time.
  template <typename Set>
  auto operator()(int device, Set set) -> decltype(set()) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;
    if (bit & done_.load(std::memory_order_acquire)) return decltype(set())(0);
    const auto status = set();
    if (status == decltype(set())(0)) done_.fetch_or(bit, std::memory_order_release);
    return status;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace ofb
