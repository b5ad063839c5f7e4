// bmxg_pdl.cuh -- programmatic dependent launches: the kernels of a step are short,
// and a normal launch begins only when the one before has drained.  A kernel
// launched with launch_after is set up while the kernel before it still runs, and
// waits at its first statement, chain_wait, until that kernel has completed and its
// writes are visible.  Rules:
//  - every thread of such a kernel calls chain_wait before anything else (a block
//    that left without it could let the next kernel start before the one before
//    has completed);
//  - what an earlier kernel of the chain writes is not read through a load the
//    compiler may move above the wait: no read-only load (__ldg, const
//    __restrict__) at an address known before it.  Read-only loads at addresses
//    that come from data read after the wait are fine, and so are those of arrays that
//    were complete before the chain's first kernel began (the list's records in the
//    list steps: a build ends a chain).
// Measured: 2000 spheres, 100 FP64 steps 1.775 -> 1.725 ms, 200 000 spheres, 100
// FP32F list steps 1.70 -> 1.66 ms, adjoint of 20 000 spheres over 40 steps (launched
// one by one) 5.10 -> 4.64 ms.  The rod kernels do not use it: their waiting
// dependents take the places of blocks that still have work (50 000 segments, 10
// FP64 steps 1.40 -> 1.60 ms).
#pragma once
#include <cuda_runtime.h>

namespace bmxg {

__device__ __forceinline__ void chain_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// kernel<<<grid, block, smem, st>>>(args...), set up before the kernel before it
// in the stream has completed.
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // (an error is the launch status the caller reads)
}

}  // namespace bmxg
