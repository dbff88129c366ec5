// Launches with programmatic stream serialization.
#pragma once

#include <cuda_runtime.h>

namespace llb {

// Launch of kernel k with programmatic stream serialization (the kernel waits
// for the previous one itself: pdl_wait_then_release).
template <class... KArgs, class... Args>
cudaError_t launch_pdl_smem(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                            Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, args...);
}
template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*k)(KArgs...), dim3 grid, dim3 block, cudaStream_t stream, Args... args) {
    return launch_pdl_smem(k, grid, block, 0, stream, args...);
}

}  // namespace llb
