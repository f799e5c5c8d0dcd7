// Shared memory that a kernel asks to be set aside, in percent of what an SM has, once a device and kernel: the preference stays with the
// function, and the call costs a microsecond.  Shared memory and L1 are one array; without the preference a kernel with dynamic
// shared memory gets about as much of it as its blocks could use, whatever its thread-local memory loses.  (A device reset drops the
// preference: the results do not depend on it.)
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <cstdint>

namespace lfd {
template <class Kernel> inline void prefer_carveout(Kernel kernel, int percent, std::atomic<uint64_t>& devices) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev > 63 || (devices.load(std::memory_order_relaxed) >> dev & 1u)) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, percent) == cudaSuccess)
        devices.fetch_or(uint64_t(1) << dev, std::memory_order_relaxed);
}
}  // namespace lfd
