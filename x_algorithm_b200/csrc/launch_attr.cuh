// What a launcher asks of the runtime once: a function attribute belongs to the kernel as loaded on the current device, so a
// process with engines on several GPUs asks on each of them, from whichever thread launches there first.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace phx {

constexpr int LAUNCH_MAX_DEVICES = 64;   // devices beyond these ask on every launch

class OncePerDevice {
 public:
  // f() (returns cudaError_t) unless it has succeeded on the current device before
  template <typename F>
  cudaError_t run(F f) {
    int dev = -1;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= LAUNCH_MAX_DEVICES) return f(dev);
    if (done_[dev].load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t r = f(dev);
    if (r == cudaSuccess) done_[dev].store(true, std::memory_order_release);
    return r;
  }

 private:
  std::atomic<bool> done_[LAUNCH_MAX_DEVICES] = {};
};

// A kernel's raised dynamic shared-memory limit: one static object per kernel and limit.
class SmemLimit {
 public:
  template <typename Kern>
  cudaError_t raise(Kern kern, int bytes) {
    return once_.run([&](int) { return cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
  }

 private:
  OncePerDevice once_;
};

}  // namespace phx
