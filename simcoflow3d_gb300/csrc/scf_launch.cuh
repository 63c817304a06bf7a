// scf_launch.cuh -- launches that overlap the end of the kernel before them.
//
// The solvers are chains of kernels of 3 to 30 us.  With a programmatic
// dependent launch a kernel's blocks are set up as soon as every block of the
// one before has left, and wait there (after_previous) until its writes are
// visible; everything a kernel does comes after that wait, so the order of
// memory accesses is that of plain launches.  Measured, plain -> this: a
// projection at 40^3 926 -> 883 us, 64^3 in FP64 2029 -> 1954, 147x93x121
// 3304 -> 3177, 256^3 13660 -> 13557; a predictor step at 128x112x96 mixed
// 3846 -> 3363, at 67x53x75 in FP64 2153 -> 1959.  The next kernel is not let
// in earlier (griddepcontrol.launch_dependents): its blocks then pile up on the
// SMs that run out of work first, which at 256^3 cost 4%.
#pragma once
#include <cuda_runtime.h>

#include <utility>

// The first statement of every kernel that launch_after starts.  (A kernel
// whose blocks did not all wait could finish before the one it follows.)
__device__ __forceinline__ void after_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// Counts a block in, by one thread after its block's results: the block that
// gets the last count may read all the others' (release of its own, acquire
// of theirs; a block barrier extends both to the other threads).
__device__ __forceinline__ unsigned count_in(unsigned *counter)
{
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
    return old;
}
