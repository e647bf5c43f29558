// eph_launch.cuh - a kernel launch that reports its own status. After kernel<<<...>>> the status has to be fetched by
// cudaGetLastError, which also reports an error that an earlier call on this thread returned to its caller already: the
// launch would be taken for failed.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace eph {

template <typename... Params, typename... Args>
inline cudaError_t launch_kernel(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                                 Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace eph
