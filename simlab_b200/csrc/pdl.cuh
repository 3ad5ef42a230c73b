// Launches with programmatic stream serialization.  Every thread of a kernel
// launched this way waits, before it touches global memory, until the kernel
// before it has completed and its writes are visible (pdl_wait); the grid's
// blocks are launched as the last blocks of that one exit instead of after a
// launch gap of 2-3 us.  Since every such kernel waits for its predecessor, a
// completed kernel implies all earlier ones; a kernel without the wait (the
// direct bulk kernel, the wall kernel on a second stream) is launched as any
// other.  Two jobs that may run side by side share one grid (k_walls_faces): a
// grid let in early that skipped the wait because its predecessor had waited
// would have no guarantee of seeing the writes of the grid before that one.
// Nor does a kernel of a step let the next grid in while it runs: a small grid's
// blocks then crowd onto the SMs that have room first and run there several at
// a time: the rotor's face kernel took 66 us instead of 26, and letting the next
// grid in at the staged bulk's last tile cost 99 us a step instead of 85
// (256x128x128 FP16, a part at rest; at the bulk's start 30 us more on
// 512x256x256).  Without the launch attribute the wait does nothing.
#pragma once
#include <cuda_runtime.h>

namespace lbm {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

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
