// pdl.cuh -- programmatic dependent launch of the kernels of a time step.
//
// A step is a chain of short kernels, each of which needs all of the one before
// it.  Launched as plain stream (or graph) successors, a kernel's blocks are
// only scheduled when the last block of the one before has left, which on a
// small grid costs more than the kernel does.  Here every kernel of the chain
// lets its successor be scheduled at once (pdl_go, first thing) and waits for
// its predecessor's completion and memory (pdl_wait) before its first access to
// anything a predecessor writes, so that launch latency, block scheduling and
// the set-up of barriers and tables run beside the predecessor.  Blocks of a
// successor only take places that the predecessor's blocks, all of them
// scheduled by then, leave free.  Every block waits, one without work too: a
// kernel whose blocks all left early would pass for its predecessors' end with
// the next one.  What a predecessor writes is read with plain loads: the
// non-coherent load is for words unwritten while the kernel lives, and the wait
// does not hold it back.  Without the launch attribute both calls do nothing.
//
// Launched early: the sweeps, the plain path's bulk updates, and the injection,
// source and gather kernels of single steps (us per step, before and after:
// 96^3 FP64 plain 54.6 and 46.4, 48^3 FP32 chunk 14.4 and 13.2, 165x150x181
// FP64 chunk 591 and 587).  Not early: an E sweep with the Drude-Lorentz pass
// beside it, whose waiting blocks would keep that pass's out (256^3: 195 ms
// against 192 ms a run), and the small kernels of a chunk, where the sweep's
// last wave then shares its SMs with them (the same run 206 ms, 150x117x98 with
// gain 28.5 against 27.4 ms).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace cps {

__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// launch of a kernel that calls pdl_wait; early: before its predecessor ends
template <typename... P, typename... A>
void launch_pdl(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = early ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace cps
