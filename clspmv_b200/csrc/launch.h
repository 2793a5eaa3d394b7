// Kernel launches of the library.
#pragma once

#include <cuda_runtime.h>

namespace csp {

// Launches a kernel that calls grid_dependency() (kernels/common.cuh) before it touches
// anything an earlier operation of the stream may write or read, with programmatic stream
// serialization: its launch and its loads of constant arrays then overlap the tail of the
// kernel before it.  In a plain stream a dependent launch otherwise starts 2 to 4 us after
// its predecessor (one B200: a period of kernel time + 0.3 us with the attribute, kernel
// time + 2..4 us without; after a copy 4.5 us against 7.7 for an empty kernel).  After
// anything but a kernel, and in a captured graph behind such nodes, it is an ordinary
// launch.  Errors are left to cudaGetLastError().
template <class... P, class... A>
void launch_chained(void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace csp
