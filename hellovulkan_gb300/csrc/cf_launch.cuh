// cf_launch.cuh — the launch helper shared by the kernels' host code.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace cfk {

// Launches `kernel`; with `overlap`, with programmatic stream serialisation
// (see grid_dependency_wait): it may be scheduled while the stream's previous
// kernel is still running.  A single view's step uses it, as do the AABBs, the
// read-back, lookup, shading and frustum culling (2 us of a call).  Batched
// passes do not: their kernels are long (64 views 106.6 us without, 109.4 with),
// and with several streams in flight (the server) CTAs launched early would
// hold SM slots while they wait.
template <typename... Params, typename... Args>
cudaError_t launch_kernel(bool overlap, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t stream, Args&&... args)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = overlap ? attr : nullptr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace cfk
