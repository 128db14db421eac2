// Dynamic shared memory that, with what the kernel declares itself (`beside`, or more), goes beyond 48 KB: a kernel may use it only where
// it has been granted.  Once per device, since the attribute is a device's, and never less than before, since a launch in another
// thread may rely on it.
#pragma once
#include <cuda_runtime_api.h>
#include <stddef.h>
#include <mutex>

#define BN_GRANT_DEVICES 64  // (a device beyond is asked each time)
struct BnGrant {  // one per kernel, static
  std::mutex lock;
  size_t bytes[BN_GRANT_DEVICES] = {};
  cudaError_t ask(const void* kernel, size_t smem, size_t beside) {
    if (smem + beside <= 48 * 1024) return cudaSuccess;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    const bool known = device >= 0 && device < BN_GRANT_DEVICES;
    std::lock_guard<std::mutex> guard(lock);
    if (known && bytes[device] >= smem) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && known) bytes[device] = smem;
    return e;
  }
};
