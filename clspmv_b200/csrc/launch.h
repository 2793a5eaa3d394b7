// Kernel launches of the library.
#pragma once

#include <cuda_runtime.h>

namespace csp {

// Launches a kernel with programmatic stream serialization: it may become resident while
// the kernel before it in the stream still runs (once every block of that one has called
// grid_dependency(), kernels/common.cuh, or left), so that its launch and its loads of
// constant arrays overlap the tail of that kernel.  The kernel has to
//   - call grid_dependency() before it touches anything that the kernel before it may still
//     write or read.  Everything older has completed by then, since that kernel waited for it
//     too.  Two kinds of kernel touch more than constant arrays before their wait:
//     xpanel_merge_kernel reads the y of rows which xpanel_kernel does not write, and the gradient
//     kernels of csp_spmv_adjoint run beside the transposed product, whose vectors they do not
//     write, and wait at their end;
//   - wait in at least one thread whatever its arguments, so that its own completion means
//     theirs;
//   - carry __restrict__ on constant arrays only.  On any other pointer it would let the compiler
//     move a load above the wait, or read through the non-coherent path.
// In a plain stream a dependent launch otherwise starts 2 to 4 us after its predecessor (one
// B200: a period of kernel time + 0.3 us with the attribute, kernel time + 2..4 us without;
// after a copy 4.5 us against 7.7 for an empty kernel).  After anything but a kernel, and in a
// captured graph behind such nodes, it is an ordinary launch.  Errors are left to
// cudaGetLastError().
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
