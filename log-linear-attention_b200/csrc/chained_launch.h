// Chained launches (programmatic dependent launch): a kernel of a call is set up while the last CTAs of the kernel before it in the stream
// finish.  Every kernel of a call is launched this way (the self-tests' are not) and begins with chain_wait(): it waits until everything before
// it in the stream is complete and visible, so nothing but the moment of the launch changes.  A short call is a dozen kernels of 3 to 20 us, with a
// microsecond or more between each two when they are launched plainly (B = 2, T = 1984, 8 heads: 229 -> 200 us a step).
//
// No kernel lets its successor start earlier (griddepcontrol.launch_dependents): waiting CTAs take shared memory and registers from the
// ones still running.  With it at the start of every kernel the level-gradient kernel of the delta rule went from 1.11 to 1.57 ms behind
// the scan (B = 4, T = 8192, 16 heads), and a Mamba-2 step from 2.20 to 2.23 ms (B = 2, T = 16384, 32 heads).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace llattn {

#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}
#endif

}  // namespace llattn
