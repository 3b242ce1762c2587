// Kernel launches with programmatic stream serialization: the kernel may be set
// up while the previous kernel of the stream ends, and its first statement
// (gridDependency in recon.cuh) waits for that one to complete. The stages of a
// frame are a chain of short dependent kernels: one 96x64 frame 77 -> 61 us a
// call, one 1438x1079 4:2:2 frame 333 -> 321 us, one 4K detail-transfer frame
// 947 -> 934 us.
#pragma once

#include <cuda_runtime.h>

namespace lgcr_b200 {

template <class... Params, class... Args>
inline cudaError_t launchAfter(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                               cudaStream_t stream, const Args &...args) {
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
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

} // namespace lgcr_b200
