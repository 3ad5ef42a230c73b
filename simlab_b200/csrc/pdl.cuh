// Launches with programmatic stream serialization.  Every kernel of a step
// lets the next kernel's grid launch as soon as its own blocks run
// (pdl_release) and, before it touches global memory, waits until the kernel
// before it has completed, memory included (pdl_wait); so the next kernel's
// blocks are resident when the last wave drains instead of starting after a
// launch gap of 2-3 us.  Since every kernel waits for its predecessor, a
// completed kernel implies all earlier ones.  Without the launch attribute
// both instructions do nothing.
#pragma once
#include <cuda_runtime.h>

namespace lbm {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// on = false: an ordinary launch (event timing between the kernels)
template <class... P, class... A>
inline cudaError_t launch_pdl(bool on, void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = on ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, (P)args...);
}

}  // namespace lbm
