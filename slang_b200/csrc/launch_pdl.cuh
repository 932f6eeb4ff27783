// Launches that overlap the end of the kernel before them on the stream (programmatic dependent launch).
//
// A kernel launched with launch_after() may start while its predecessor is still running, so it calls grid_wait() before
// its first access to global memory; that returns when the predecessor has completed and its writes are visible.  Because
// every such kernel waits before it completes, completion stays in stream order.  grid_release() lets the successor's
// blocks start as soon as every block of this kernel has been placed; they hold no work back, they only wait.
//
// Tensor memory is taken after grid_wait() and the successor released after that, by the warp that took it (one thread's
// release counts for its block).  A block that held tensor memory while it waits could keep a block of its predecessor on
// the same SM from ever getting its own, and a block that has yet to take some must not let in a successor that does so first.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace mlpb200 {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A kernel's dynamic shared-memory limit, raised once per device instead of on every launch (one static object per kernel;
// the attribute outlives the call, and raising it twice from two threads does no harm).
struct SmemLimit {
    std::atomic<uint64_t> raised{0};   // bit d: device d
    cudaError_t raise(const void* kernel, int device, size_t bytes)
    {
        const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;
        if (raised.load(std::memory_order_relaxed) & bit) return cudaSuccess;
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e == cudaSuccess) raised.fetch_or(bit, std::memory_order_relaxed);
        return e;
    }
};

template <class... P, class... A>
inline cudaError_t launch_after(cudaStream_t st, void (*kernel)(P...), uint32_t grid, uint32_t block, size_t smem, A&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace mlpb200
