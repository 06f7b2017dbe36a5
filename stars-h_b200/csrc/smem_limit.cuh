// Dynamic shared-memory limits of kernels.  What a launch may ask for above
// 48 KB is one number per function and device, the same for every host thread
// of the process.  A limit set before each launch, to what that launch needs,
// can therefore be lowered by another thread (a call's second lane, a serving
// worker) between the setting and the launch, which then fails.  So a kernel's
// limit is set once per device, to the most any of its launches asks for.
#pragma once
#include <atomic>
#include <cuda_runtime.h>

namespace b200 {

// Allows launches of Kernel with up to Bytes of dynamic shared memory on the
// current device.  Bytes is a compile-time bound over all launches of Kernel:
// threads that get here together set the same number.
template <auto Kernel, size_t Bytes>
inline cudaError_t allow_smem()
{
    static std::atomic<unsigned long long> devices{0};   // of the first 64
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (devices.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute((const void *)Kernel,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Bytes);
    if (e == cudaSuccess) devices.fetch_or(bit, std::memory_order_release);
    return e;
}

// Streaming multiprocessors of the current device (148 if it does not say).
inline int sm_count()
{
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        n <= 0)
        return 148;
    return n;
}

}  // namespace b200
