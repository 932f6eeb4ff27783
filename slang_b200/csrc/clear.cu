// Clears of a few words (a loss buffer).  A kernel, because a kernel overlaps its neighbours on the stream and a memset does
// not: in a queue of steps the example's takes 7.5 us, 8.2 with a memset, 4096 samples of 2-16-16-16-1 13.5 and 14.3; a single step gains nothing, as a launch costs the
// host 3.7 us and a memset 1.2.  In a unit of its own, so that a
// program's first clear loads no other kernels.
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch_pdl.cuh"
#include "launchers.h"

namespace mlpb200 {

__global__ void __launch_bounds__(256) clear_bytes_kernel(uint8_t* p, uint32_t size)
{
    grid_release();
    grid_wait();
    if ((((uint64_t)p | size) & 3u) == 0) {
        for (uint32_t i = threadIdx.x; i < size / 4; i += 256) ((uint32_t*)p)[i] = 0u;
    } else {
        for (uint32_t i = threadIdx.x; i < size; i += 256) p[i] = 0;
    }
}

cudaError_t launch_clear_bytes(cudaStream_t st, void* p, uint32_t size) { return launch_after(st, clear_bytes_kernel, 1, 256, 0, (uint8_t*)p, size); }

}  // namespace mlpb200
