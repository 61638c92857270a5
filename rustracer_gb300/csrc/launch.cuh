// launch.cuh — chains of short kernels whose launches overlap (programmatic
// dependent launch).  A kernel launched by launch_after is brought up while the
// one before it in the stream still runs, and waits in after_previous(), its
// first statement, until that one is complete; so the gap between two kernels,
// 1 to 2 us of the 5 to 10 that one of a small frame or a build's later rounds
// takes, shrinks to the wait's return.  A block that waits holds only room that
// the earlier kernel no longer asks for: the next one is let in when all its
// blocks have started.  Across an event, a copy or a memset the order is the
// stream's own.  Cornell box of 64 x 64 paths 181 -> 164 us, of 512 x 512
// 357 -> 330; material zoo at 854 x 480 and 3 samples 1,841 -> 1,818.
#pragma once
#include <cuda_runtime.h>

#include "vec.cuh"

namespace gbrt {

// What ran before this kernel in its stream is complete and visible from here on.
GB_D void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launches a kernel that begins with after_previous().
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), uint32_t blocks, uint32_t threads, cudaStream_t stream,
                         const A&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace gbrt
