// Launching a kernel behind the one before it in a stream (internal to the library).
#pragma once

#include <cuda_runtime.h>

namespace nbody {

// Launches `kernel` so that its launch overlaps the end of the kernel before it
// in the stream (programmatic dependent launch). The kernel begins with
// wait_for_launches_before(), so it sees a finished predecessor all the same;
// what goes away is the gap between the two, 1 to 2 us. Forces of 30,001 bodies
// (14 launches): 184 -> 161 us; a host step of 4,096: 170 -> 167; ten resident
// steps of 262,144: 11.41 -> 11.36 ms (GB300). Every kernel launched this way
// waits in all its threads before it reads or writes memory, so a chain of them
// is as ordered as plain launches (but for walks side by side: bh.h).
template <class... Params, class... Args>
cudaError_t launch_behind(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                          Args &&...args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace nbody
