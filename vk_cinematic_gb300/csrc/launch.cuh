// Chained kernel launches.
#pragma once

#include <cuda_runtime.h>

namespace gbsp {

// Kernels that follow one another through memory.  Launched with
// launch_next, a kernel may become resident while the one before it drains;
// stage_begin, its first statement, holds it until that one has completed and
// its writes are visible, and only then lets the next one in.  The chain is
// transitive: a kernel completes after its predecessor did.  What one of them
// writes, the next reads by plain loads: no __ldg and no const __restrict__,
// which promise data that is constant for the whole life of a kernel.
// A kernel that lets the next one in early writes nothing that the next one
// reads before its own stage_begin (weights, tables).
// 128 x 128 x 8 frame 227 -> 214 us, 641 x 359 x 7 watertight 929 -> 899 us, a
// 128 x 128 x 4 crop 248 -> 232 us; long kernels are the same either way.
__device__ __forceinline__ void stage_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// For kernels that call stage_begin before they touch memory that others write.
template <class... P, class... A>
void launch_next_smem(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, const A &...args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);  // the caller reads cudaGetLastError
}

template <class... P, class... A>
void launch_next(void (*kernel)(P...), int grid, int block, cudaStream_t s, const A &...args)
{
    launch_next_smem(kernel, grid, block, 0, s, args...);
}

}  // namespace gbsp
