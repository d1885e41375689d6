// mpm_launch.cuh -- kernel launches of a chain: each kernel's CTAs may start
// while the last ones of the kernel before it end (programmatic stream
// serialization); the kernel waits for that one's results with follow().
#pragma once

#include <cuda_runtime.h>

namespace mpm {

template <class... Args>
cudaError_t launch_following(cudaStream_t stream, void (*kernel)(Args...), dim3 grid, dim3 block, size_t shared,
                             Args... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = shared;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace mpm
