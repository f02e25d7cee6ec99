// Dynamic shared memory past 48 KB, which every kernel has to be allowed on every device it runs on.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstddef>

namespace avd {

// Allows `Kernel` up to `bytes` of dynamic shared memory on the current device. The attribute is the
// device's, so a process that runs engines on two devices sets it on both: a bit per device remembers
// where it is set (a query of the current device costs far less than setting it again). One kernel takes
// one `bytes` for all its callers. Devices past the word's bits set it every time; a failure is not
// remembered.
template <auto Kernel>
cudaError_t allow_smem(size_t bytes) {
    static std::atomic<unsigned long long> allowed{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (allowed.load(std::memory_order_relaxed) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute(reinterpret_cast<const void*>(Kernel), cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(bytes));
    if (e == cudaSuccess) allowed.fetch_or(bit, std::memory_order_relaxed);
    return e;
}

}  // namespace avd
