// per_context.h — set-up that a kernel needs once in every device context it runs in.
//
// The shared memory a kernel may ask for above 48 KB, and cluster sizes above 8, are
// attributes that cudaFuncSetAttribute gives to the kernel in the current device's
// context: a process that has set them on one device has not on another, nor on the same
// one after cudaDeviceReset.  Plain C++ (the CUDA calls are the caller's).
#pragma once

#include <atomic>

namespace vpm {

constexpr int kMaxDevices = 64;

class PerContext {
 public:
  // set() -> 0 when it succeeded, run unless it has succeeded before in context `ctx` (the
  // id of the current context, 0 when unknown) of device `dev`.  Threads may run it
  // twice; it sets the same values each time.
  template <class Set>
  int ensure(int dev, unsigned long long ctx, Set set) {
    const bool known = dev >= 0 && dev < kMaxDevices && ctx != 0;
    if (known && done_[dev].load(std::memory_order_acquire) == ctx) return 0;
    const int e = set();
    if (e == 0 && known) done_[dev].store(ctx, std::memory_order_release);
    return e;
  }

 private:
  std::atomic<unsigned long long> done_[kMaxDevices] = {};
};

}  // namespace vpm
