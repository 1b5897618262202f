// Launch helpers of the kernels that follow one another on a stream.
//
// A Lanczos step of a small sector is a kernel of a few microseconds, most of
// which are its launch and the chain of loads before the first element: the
// launches are programmatic (the next kernel's blocks start while the previous
// grid drains and stage what no earlier kernel writes -- tables, palettes,
// coefficients -- before they wait for it), and what a launch asks the runtime
// about a kernel is asked once per thread, kernel and block shape.  H*v of a
// sector of 400 or 4,900 states called in a row: 6.1 us a call, 3.6 us now (the
// host's part of a call).  A fused step of a 160-step chain, two-step graphs
// before, programmatic launches with the first row group's tables ahead of the
// wait now: 400 states 10.3 -> 6.6 us, 15,876 12.3 -> 8.0, 853,776 26.5 -> 21.8,
// 2,944,656 55.7 -> 50.6.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace edk {

// Everything the kernels before this one wrote is visible after it, and they
// have ended.  Every block of a kernel launched with launch_chained calls it,
// before it reads or writes anything another kernel may write or read.  What another
// kernel of the chain wrote is read with ordinary loads or ld.cg, not through the
// read-only path and not through const __restrict__ pointers.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel may start its blocks once all of this one's have come here.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Allows `kernel` the dynamic shared memory `smem` and gives the blocks of
// `threads` threads that an SM holds.  The limit belongs to the process: it is set
// to all the kernel can have, never to one call's need, which another thread's
// smaller call could lower between this one's setting and its launch.
cudaError_t kernel_fit(const void *kernel, int threads, size_t smem, int *per_sm);

template <typename... K, typename... A>
cudaError_t launch_chained(void (*kernel)(K...), int grid, int block, size_t smem, cudaStream_t st, const A &...args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, K(args)...);
}

}  // namespace edk
