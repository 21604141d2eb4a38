// What a launch asks a device once: the opt-in to more shared memory than 48 KB, the number of SMs.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

namespace kb2 {

// cudaFuncAttributeMaxDynamicSharedMemorySize is a PER-DEVICE attribute: one process may drive several GPUs (the
// reference's EP layout, python/krasis/model.py:1496-1523), so the opt-in is remembered per device ordinal, not per
// process.  Thread-safe (atomic flags; setting the attribute twice is harmless).
struct PerDeviceOnce {
  std::atomic<bool> done[64];
  PerDeviceOnce() { for (auto& d : done) d.store(false); }
  // returns the current device ordinal if its opt-in is still pending, else -1
  int pending() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;   // unknown device: always (re)configure
    return done[dev].load(std::memory_order_acquire) ? -1 : dev;
  }
  void mark(int dev) { if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release); }
};

// SMs of the current device
inline int current_sms() {
  static std::atomic<int> known[64];
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if ((sms = known[dev].load(std::memory_order_relaxed)) > 0) return sms;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 148;
  known[dev].store(sms, std::memory_order_relaxed);
  return sms;
}

// The opt-in of kKernel to `bytes` of dynamic shared memory, the most that any of its launches takes: a size that followed from a call's arguments
// could be lowered by another thread between a call's opt-in and its launch.
template <auto kKernel>
inline cudaError_t allow_smem(int bytes) {
  static PerDeviceOnce once;
  const int dev = once.pending();
  if (dev < 0) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) once.mark(dev);
  return e;
}

}  // namespace kb2
