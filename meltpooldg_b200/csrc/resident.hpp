// What a kernel may use on a device: its limit of dynamic shared memory and the CTAs that are
// resident at once. Both belong to the kernel on one device, so they are set and asked once per
// device and not once per process. One static object per kernel; safe with several threads.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include <atomic>
#include <mutex>

namespace mpdg {

constexpr int kMaxDevices = 64;

inline cudaError_t current_device(int *device)
{
  const cudaError_t e = cudaGetDevice(device);
  if (e != cudaSuccess) return e;
  return *device >= 0 && *device < kMaxDevices ? cudaSuccess : cudaErrorInvalidDevice;
}

// The limit of dynamic shared memory (48 KB by default), raised to the largest size asked for.
class SharedLimit {
 public:
  template <typename K> cudaError_t raise(K kernel, size_t bytes)
  {
    int device = 0;
    cudaError_t e = current_device(&device);
    if (e != cudaSuccess || bytes <= limit_[device].load(std::memory_order_acquire)) return e;
    std::lock_guard<std::mutex> lock(mu_);
    if (bytes <= limit_[device].load(std::memory_order_relaxed)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) limit_[device].store(bytes, std::memory_order_release);
    return e;
  }

 private:
  std::mutex mu_;
  std::atomic<size_t> limit_[kMaxDevices] = {};
};

// The CTAs of a kernel at one launch shape that the current device holds at once.
class ResidentBlocks {
 public:
  template <typename K> cudaError_t get(K kernel, int threads, size_t smem, int *blocks)
  {
    int device = 0;
    cudaError_t e = current_device(&device);
    if (e != cudaSuccess) return e;
    int b = blocks_[device].load(std::memory_order_acquire);
    if (b == 0) {
      int per_sm = 0, sms = 0;
      if (smem > 48 * 1024)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
      if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
      if (e != cudaSuccess) return e;
      b = per_sm * sms;
      if (b < 1) return cudaErrorLaunchOutOfResources;
      blocks_[device].store(b, std::memory_order_release);
    }
    *blocks = b;
    return cudaSuccess;
  }

 private:
  std::atomic<int> blocks_[kMaxDevices] = {};
};

}  // namespace mpdg
