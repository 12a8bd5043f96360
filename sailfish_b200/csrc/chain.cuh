// Launches chained with programmatic dependent launch. A step is a chain of
// four to six kernels on one stream, each reading what the one before wrote;
// on small grids the gaps between them are a quarter of the step. A chained
// kernel is scheduled while its predecessor still runs and waits on the
// device for it to finish and its writes to be visible.
//
// Every chained kernel calls chain_begin() in all threads before it touches
// global memory, so it never starts work before all kernels ahead of it on
// the stream have finished (its predecessor waited for its own). Launched any
// other way, or behind a kernel that does not take part, that does nothing.
// The successor is let in by chain_end() (or the block's exit) when the
// block's work is done: it is scheduled once every block has come that far,
// onto SMs that are about to be empty. Let in at the beginning instead, its
// blocks were spread over whatever slots the running kernel had left, and
// the imbalance cost more than the gap (512^2: 65 us a step without chaining,
// 78 with an early, 60 with a late successor).
#pragma once

#include <cuda_runtime.h>

namespace cbd {

__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

__device__ __forceinline__ void chain_end() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// A launch that fails leaves no error behind for a later call to find (the
// other entry points ask for the last error after their launches).
template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args)
{
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
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    if (e != cudaSuccess)
        cudaGetLastError();
    return e;
}

}  // namespace cbd
