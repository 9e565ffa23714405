// What has to be done once on every device of a process, such as raising a kernel's limit of dynamic shared
// memory: the attribute belongs to the device that is current when it is set, so once in a process is not enough.
#pragma once
#include <atomic>
#include <cstdint>

namespace amem {

// A bit per device; devices beyond 64 are done every time.  Two threads may both do it (what is done is the same
// twice over); a failure leaves the bit unset, so the next call tries again.
class OncePerDevice {
 public:
  template <typename F>   // F: () -> error code, 0 for success
  auto operator()(int device, F&& what) -> decltype(what()) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
    if (bit && (done_.load(std::memory_order_acquire) & bit)) return decltype(what())(0);
    const auto e = what();
    if (e == decltype(what())(0) && bit) done_.fetch_or(bit, std::memory_order_acq_rel);
    return e;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace amem
