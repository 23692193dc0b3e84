// Internal: what the launchers of the library's kernels share.
#ifndef SAL_LAUNCH_H
#define SAL_LAUNCH_H

#include <cuda_runtime.h>

#include <atomic>

// Lets `kernel` be launched with all the dynamic shared memory that the current device gives a block.  The limit belongs to the (kernel,
// device) pair and is set once, to its largest value: one that followed the launches' needs could be lowered by a thread with a smaller
// launch between another thread's look at it and its launch.  `done` is the kernel's own, per device ordinal.
template <typename Kernel>
cudaError_t sal_allow_shared_memory(Kernel *kernel, std::atomic<bool> (&done)[64]) {
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (done[dev].load(std::memory_order_acquire)) return cudaSuccess;
    cudaFuncAttributes attr;
    if ((e = cudaFuncGetAttributes(&attr, kernel)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)attr.sharedSizeBytes)) != cudaSuccess) return e;
    done[dev].store(true, std::memory_order_release);
    return cudaSuccess;
}

#endif
