// Launches with programmatic stream serialization.  Every kernel of a step
// waits, before it touches global memory, until the kernel before it has
// completed, memory included (pdl_wait), and its blocks are launched as the
// last blocks of that one exit instead of after a launch gap of 2-3 us.  Since
// every kernel waits for its predecessor, a completed kernel implies all
// earlier ones.  pdl_release lets the next grid in earlier; only the wall
// kernel uses it, for the face kernel that runs beside it.  Let in while a
// kernel runs, a small grid's blocks crowd onto the SMs that have room first
// and run there several at a time: the rotor's face kernel took 66 us instead
// of 26, and letting the next grid in at the staged bulk's last tile cost 99 us
// a step instead of 85 (256x128x128 FP16, a part at rest; at the bulk's start
// 30 us more on 512x256x256).  Without the launch attribute both instructions
// do nothing.
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
