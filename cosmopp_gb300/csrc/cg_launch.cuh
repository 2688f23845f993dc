// Launches that overlap the end of the kernel before them in the stream.
#pragma once

#include <cuda_runtime.h>

#include "cg_internal.h"

namespace cg {

// Programmatic dependent launch: the next kernel of the stream may take its place as soon as SMs are free
// and does its set-up there; what it reads and writes comes after the wait for this one.  A kernel boundary
// took 4 us without it.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_prior() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// a launch that may start beside the end of the kernel before it (launch_dependents, wait_prior), in clusters
// of `cluster` CTAs
template <typename... P, typename... A>
static int launch(cg_ctx* ctx, void (*kernel)(P...), dim3 grid, int threads, size_t smem, int cluster, cudaStream_t s,
                  A... args)
{
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = cluster;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    count_launch(ctx);
    CG_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, kernel, P(args)...));
    return CG_OK;
}

}  // namespace cg
