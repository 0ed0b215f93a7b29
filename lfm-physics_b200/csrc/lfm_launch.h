// Raising a kernel's limit of dynamic shared memory.
#pragma once

#include <mutex>

#include <cuda_runtime.h>

namespace lfm {

// The limit is an attribute of (kernel, device): a process that steps lattices on two
// GPUs has to raise it on each.  One object a kernel remembers what it raised where.
class SmemGrant {
 public:
  // Lets `kernel` take `smem` bytes of dynamic shared memory on the current device;
  // cudaErrorNotSupported where the device has no room for them beside the kernel's
  // static ones.
  cudaError_t raise(const void* kernel, int smem) {
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu_);
    const bool kept = dev >= 0 && dev < kDevices;
    if (kept && smem <= granted_[dev]) return cudaSuccess;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa{};
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    if (smem + (int)fa.sharedSizeBytes > optin) return cudaErrorNotSupported;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess && kept) granted_[dev] = smem;
    return e;
  }

 private:
  static constexpr int kDevices = 64;
  std::mutex mu_;
  int granted_[kDevices] = {};
};

}  // namespace lfm
