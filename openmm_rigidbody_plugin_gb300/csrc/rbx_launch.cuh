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

constexpr size_t kSharedPerSM = 228 * 1024;  // the most that an SM of GB300 sets aside

template <class T> struct as_is { using type = T; };

// `shared` > 0: shared memory to set aside per SM, in bytes (a preference); the rest is L1.
template <class... A>
cudaError_t launch_chained_l1(size_t shared, void (*kernel)(A...), int grid, int block, size_t smem, cudaStream_t st,
                              typename as_is<A>::type... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (shared) {
        const size_t percent = (100 * shared + kSharedPerSM - 1) / kSharedPerSM;
        attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        attr[1].val.sharedMemCarveout = percent < 100 ? (unsigned)percent : 100u;
        cfg.numAttrs = 2;
    }
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <class... A>
cudaError_t launch_chained(void (*kernel)(A...), int grid, int block, size_t smem, cudaStream_t st,
                           typename as_is<A>::type... args) {
    return launch_chained_l1<A...>(0, kernel, grid, block, smem, st, args...);
}

}  // namespace rbx
