// launch.cuh -- launches whose start overlaps the end of the kernel before them (programmatic dependent launch), and the
// step index that a stretch of launches shares.
//
// A kernel launched by launch_after() may start while its predecessor in the stream still runs; it sets itself up, then
// calls wait_predecessor(), which returns once the predecessor has completed and its writes are visible. It then calls
// allow_successor(), so that the kernel after it may start in turn: because every kernel waits before it lets the next one
// start, a kernel that has started knows that everything before its direct predecessor is complete. Nothing that the
// direct predecessor writes may be touched before the wait. An ordinary load through a __restrict__ pointer could be moved
// above it by the compiler, which sees no write to that memory: what a predecessor writes is read by volatile loads (copies
// to shared memory, ld_cg) or through pointers that may alias.
#pragma once

#include <cuda_runtime.h>

#include "engine.h"

__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_successor() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    g_launches++;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// A plane launch that is given a counter advances its Philox step index once every CTA has read it: the CTA that finishes
// last (the counter reaches the grid size) resets the counter and adds sr.inc.
__device__ __forceinline__ void advance_step(const StepRef &sr)
{
    if (!sr.done) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(sr.done, 1) == (int)gridDim.x - 1) {
            *sr.done = 0;
            atomicAdd(sr.step, sr.inc);
        }
    }
}
