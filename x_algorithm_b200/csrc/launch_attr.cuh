// What a launcher asks of the runtime once: a function attribute belongs to the kernel as loaded on the current device, so a
// process with engines on several GPUs asks on each of them, from whichever thread launches there first.
#pragma once
#include <cuda_runtime.h>

#include <stdlib.h>
#include <string.h>

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

// Launch of a kernel that waits (griddepcontrol.wait) before it touches memory: it may set up, and fill SMs as they come free,
// while the kernel in front of it on the stream finishes.  PHX_PDL=0 keeps plain stream order.
template <typename... P, typename... A>
cudaError_t launch_programmatic(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = grid; lc.blockDim = block; lc.dynamicSmemBytes = smem; lc.stream = stream;
  cudaLaunchAttribute at[1];
  static const bool pdl = !(getenv("PHX_PDL") && getenv("PHX_PDL")[0] == '0');
  if (pdl) {
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at; lc.numAttrs = 1;
  }
  return cudaLaunchKernelEx(&lc, kern, static_cast<P>(args)...);
}

// SMs of the current device
inline int device_sms() {
  static std::atomic<int> known[LAUNCH_MAX_DEVICES] = {};
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 148;
  const bool kept = dev >= 0 && dev < LAUNCH_MAX_DEVICES;
  if (kept && (n = known[dev].load(std::memory_order_relaxed)) > 0) return n;
  if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
  if (kept) known[dev].store(n, std::memory_order_relaxed);
  return n;
}

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
