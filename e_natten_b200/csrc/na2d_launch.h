// Launches that overlap the end of the kernel before them in the stream.
#pragma once

#include <cuda_runtime.h>

namespace na2d_launch {

// Launches a kernel that calls na2d_ptx::after_previous_grid() before it touches what kernels write.  `overlap`: its blocks may start once the
// kernel before it in the stream lets them (na2d_ptx::next_grid_may_start; any other kernel does by ending), and set themselves up while
// the last blocks of that one run.
template <typename... P, typename... A>
cudaError_t launch(bool overlap, void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = st;
    config.attrs = &attribute;
    config.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
    return cudaGetLastError();
}

}  // namespace na2d_launch
