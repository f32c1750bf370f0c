// Launches that overlap their own start with the end of the kernel before them (programmatic dependent launch).
//
// A kernel launched by LaunchChained is set up, and its first CTAs are put on the SMs, while the last CTAs of its
// predecessor in the stream drain.  It must call WaitForPrevious before it touches any memory: that returns when the
// predecessor has completed and its writes are visible, so what the caller sees is the usual stream order; only the
// launch latency and the ramp-up are hidden.  A predecessor that is not a kernel (a copy, a memset) is waited for as
// always.  Back-to-back products of a 4096-row matrix: 4.1 us apart with ordinary launches, 2.5 us (what the host takes to
// issue one) with these; 2 entries in each of 805,575 rows: 16.4 and 10.4 us.
// No kernel gives the next one leave to start earlier (griddepcontrol.launch_dependents): the waiting CTAs then hold the
// slots that the CTAs of a grid of several waves are about to take (14.0 us on the second example, and 16.3 instead of
// 11.2 us on 27,197 rows of which 300 are long).
#pragma once

#include <utility>

#include <cuda_runtime.h>

namespace b200sp {

__device__ __forceinline__ void WaitForPrevious() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
inline cudaError_t LaunchChained(void (*kernel)(Params...), unsigned grid, unsigned threads, size_t smem, cudaStream_t stream,
                                 Args &&...args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(std::forward<Args>(args))...);
}

}  // namespace b200sp
