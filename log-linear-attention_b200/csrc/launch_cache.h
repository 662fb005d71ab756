// Host-side facts that a launch needs and that do not change: asked of the runtime once per thread and device instead of on every
// launch (an attribute call costs about as much as a launch's own argument marshalling).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <initializer_list>

namespace llattn {

// Whether one of the pointers (a null one is not) does not start on a multiple of `bytes`: vector loads and stores there would fault.
inline bool misaligned(size_t bytes, std::initializer_list<const void*> ptrs) {
    for (const void* p : ptrs)
        if (reinterpret_cast<uintptr_t>(p) % bytes != 0) return true;
    return false;
}

// The kernel may use `bytes` of dynamic shared memory on the current device.
inline cudaError_t allow_smem_of(const void* fn, size_t bytes) {
    struct Entry {
        const void* fn;
        int dev;
        size_t bytes;
    };
    static thread_local Entry table[256] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    Entry& t = table[((reinterpret_cast<uintptr_t>(fn) >> 4) * 31 + dev) & 255];
    if (t.fn == fn && t.dev == dev && t.bytes == bytes) return cudaSuccess;
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) t = Entry{fn, dev, bytes};
    return e;
}
template <typename KernT>
inline cudaError_t allow_smem(KernT kern, size_t bytes) {
    return allow_smem_of(reinterpret_cast<const void*>(kern), bytes);
}

inline cudaError_t sm_count(int* sms, int dev) {
    static thread_local int count[64] = {};
    if (dev >= 0 && dev < 64 && count[dev] > 0) {
        *sms = count[dev];
        return cudaSuccess;
    }
    const cudaError_t e = cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess && dev >= 0 && dev < 64) count[dev] = *sms;
    return e;
}

}  // namespace llattn
