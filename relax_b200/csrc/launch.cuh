// launch.cuh -- launch helpers shared by the translation units.
#pragma once

#include <cuda_runtime.h>

template <typename K>
static void set_smem(K kern, size_t sm)
{
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
}

// A launch with programmatic dependent launch allowed: the kernel (one that
// enters through pdl_enter) may be scheduled while the previous kernel in the
// stream finishes its last wave, and waits for it before touching memory.
// Errors are left for cudaGetLastError, as with <<< >>>.
template <typename... P, typename... A>
static void launch_pdl(void (*kern)(P...), dim3 grid, dim3 block, size_t sm, cudaStream_t st, const A &...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = sm;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kern, args...);
}
