// The shared memory that a kernel's launches may ask for above the usual 48 KB.  The driver keeps that limit for each kernel on
// each device, so a launcher that does not set it anew for every launch keeps in mind how much it has set on which device: a
// static OptIn for a kernel, or for several of the same need, called before a launch on the current device.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <atomic>
#include <initializer_list>
#include <mutex>

namespace pbe {

class OptIn {
 public:
  template <typename... Kernels>
  cudaError_t operator()(size_t bytes, Kernels*... kernels) {
    int device = 0;
    const cudaError_t rc = cudaGetDevice(&device);
    if (rc != cudaSuccess) return rc;
    const bool kept = device < DEVICES;                  // devices from there on are set before every launch
    if (kept && most_[device].load(std::memory_order_acquire) >= bytes) return cudaSuccess;
    std::lock_guard<std::mutex> lock(setting_);
    if (kept && most_[device].load(std::memory_order_relaxed) >= bytes) return cudaSuccess;
    for (const cudaError_t e : {cudaFuncSetAttribute(kernels, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)...})
      if (e != cudaSuccess) return e;
    if (kept) most_[device].store(bytes, std::memory_order_release);
    return cudaSuccess;
  }

 private:
  static constexpr int DEVICES = 16;
  std::atomic<size_t> most_[DEVICES] = {};
  std::mutex setting_;
};

}  // namespace pbe
