// Launches that overlap the end of the launch before them.
#pragma once

#include <cuda_runtime.h>

namespace sw {

// A run is a chain of launches, and a launch that starts when the one before it
// has drained costs 4 us whatever it does.  launch_dependent lets a
// launch be scheduled earlier (programmatic dependent launch); it waits here,
// before its first access, for the previous one to have completed and its
// writes to be visible: 1.6 us per launch on small domains.  The previous
// kernel's blocks release it as they exit, not before: released at their start,
// its blocks settled on SMs still at work and left others idle (KS FP64, 65536
// cells: 4.9 ms for 600 launches, 1.8 as it is, 3.6 without any of this).
//
// A kernel that waits here, and every device function it calls, takes the
// pointers that the previous launch may have written without __restrict__: that
// would declare their memory unchanged for the kernel's whole life, which begins
// before the wait, and allow reads through the read-only path or above the wait.
// What is read before the wait (the closure's staged weights) was written by an
// ordinary launch in front of the whole chain.
__device__ __forceinline__ void wait_for_previous_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A launch that may be scheduled while the launch before it drains
// (wait_for_previous_launch).  Its error is returned and not left behind as the
// thread's last one, which the end of the next run would report again.
template <typename... K, typename... A>
cudaError_t launch_dependent(void (*kernel)(K...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, K(args)...);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace sw
