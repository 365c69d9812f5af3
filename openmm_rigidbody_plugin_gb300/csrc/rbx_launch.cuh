// rbx_launch.cuh -- chained kernel launches: a kernel of a chain may be scheduled while the kernel before
// it in its stream drains (programmatic dependent launch), so that its launch latency and the loads of
// its constant tables overlap that kernel's tail.
//
// Every chained kernel calls chain_release() first (the next kernel may be scheduled once all blocks
// have) and chain_wait() before it touches anything that an earlier kernel writes, in every thread and on
// every path: the wait returns when the kernel before has completed and its writes are visible, and
// that kernel waited likewise, so order along the stream is kept. Before the wait only tables that the
// host set up under a synchronisation are read. Data written by earlier kernels is never read through
// the read-only (__ldg) path, whose loads the compiler may move above the wait.
#pragma once

#include <cuda_runtime.h>

namespace rbx {

__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class T> struct as_is { using type = T; };

template <class... A>
cudaError_t launch_chained(void (*kernel)(A...), int grid, int block, size_t smem, cudaStream_t st,
                           typename as_is<A>::type... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace rbx
