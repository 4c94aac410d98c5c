// shared_memory.hpp — a kernel's opt-in to more dynamic shared memory than the default 48 KB.
#pragma once
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdint>

namespace wlg {

// The attribute belongs to the kernel on one device: it is set once on each, and the record of that may be
// read and written by several host threads (whoever finds the bit has the attribute set).
class SharedMemoryOptIn {
  public:
    cudaError_t operator()(const void* kernel) {
        int device = 0;
        cudaError_t status = cudaGetDevice(&device);
        if (status != cudaSuccess) return status;
        const uint64_t bit = device < 64 ? uint64_t{1} << device : 0;
        if (done_.load(std::memory_order_acquire) & bit) return cudaSuccess;
        status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (status == cudaSuccess) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }

  private:
    std::atomic<uint64_t> done_{0};
};

}  // namespace wlg
