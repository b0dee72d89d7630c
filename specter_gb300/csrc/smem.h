// Opting in to more shared memory a block than the 48 KB that every kernel has.
#pragma once

#include <map>
#include <mutex>

#include <cuda_runtime.h>

namespace sg {

// The dynamic shared memory that a kernel can be given: 227 KB without its static arrays.
inline int smem_most(const void *kernel) {
    static std::mutex lock;
    static std::map<const void *, int> most;
    std::lock_guard<std::mutex> hold(lock);
    int &m = most[kernel];
    if (!m) {
        cudaFuncAttributes a{};
        if (cudaFuncGetAttributes(&a, kernel) != cudaSuccess) return 0;
        m = 227 * 1024 - (int)a.sharedSizeBytes;
    }
    return m;
}

// Before a launch with `bytes` of dynamic shared memory.  The limit belongs to the kernel and all threads of
// the process share it, so it is always the kernel's largest: were it this launch's, a plan of another length
// on another thread could lower it before the launch.  (40 KB: kernels with static arrays opt in early.)
template <typename K>
void allow_smem(K kernel, size_t bytes) {
    if (bytes > 40 * 1024)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_most((const void *)kernel));
}

}  // namespace sg
