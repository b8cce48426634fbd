// chain.cuh — kernels launched before the one ahead of them in the stream ends.
//
// A kernel launched with launch_chained() may be brought up while the kernel
// directly ahead of it in the stream still runs its last blocks.  Both begin with
// chain_begin(), which waits until everything ahead has finished and its writes
// are visible, and then lets the next one be brought up in turn: nothing a kernel
// reads or writes moves ahead of its stream order, whatever ran before it.
//
// What it saves is the gap between two launches, 1 to 2 us.  It is used where it
// measured faster: shading behind the hit split and the counter reset behind the
// shadow rays (160 x 120 preview 638 -> 592 us, 256^2 at 16 spp 1585 -> 1550),
// and the denoiser's convolutions, weight and bias gradients (forward at
// 1080 x 1920 1021 -> 993 us, gradients at 16 x 256 x 256 2217 -> 2132).  Not for the
// closest-hit kernel: its blocks would wait in the slots that the shadow rays'
// could run in (333 x 217 with textures 1015 -> 1080 us); not behind a wait for
// another stream (the hit split: 256^2 1585 -> 1675 us); and not for pooling and
// upsampling (forward 1021 -> 1042 us).
#pragma once

#include <cuda_runtime.h>

namespace pt {

// Before anything else, by all threads.
__device__ __forceinline__ void chain_begin()
{
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

// Only for kernels that begin with chain_begin().
template <class... Params, class... Args>
void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, Params(args)...); // cudaGetLastError returns its error
}

} // namespace pt
