// A kernel's limit on dynamic shared memory is an attribute of the kernel on one device: it has to be raised once on
// each device that launches the kernel, whatever number of devices one process drives.
#pragma once

#include <cuda_runtime.h>

#include <atomic>

namespace sageb200 {

// One static object per kernel.  Raises the limit on the current device unless that has been done; devices past the
// table are asked each time.
class SharedOptIn {
 public:
  cudaError_t operator()(const void *kernel, size_t bytes) {
    int device = 0;
    cudaError_t error = cudaGetDevice(&device);
    const bool kept = device >= 0 && device < kDevices;
    if (error == cudaSuccess && !(kept && done_[device].load(std::memory_order_acquire))) {
      error = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
      if (error == cudaSuccess && kept) done_[device].store(true, std::memory_order_release);
    }
    if (error != cudaSuccess) cudaGetLastError();  // (reported to the caller, not left for the next launch)
    return error;
  }

 private:
  static constexpr int kDevices = 64;
  std::atomic<bool> done_[kDevices] = {};
};

}  // namespace sageb200
