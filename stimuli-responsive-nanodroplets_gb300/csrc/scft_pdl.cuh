/*
 * scft_pdl.cuh — launches that overlap the end of the kernel before them
 * (programmatic dependent launch): a CTA may start once every CTA of the kernel
 * before has triggered or ended, and pdl_wait() returns when that kernel, and all
 * it waited for itself, is complete. Every CTA of such a kernel calls pdl_wait()
 * on every path, so that kernels complete in stream order, and touches nothing
 * that a kernel writes before it; nor does it read such data by the read-only path
 * (__ldg), which takes them as constant from the kernel's start on. The tensor-core passes load their operator
 * digits meanwhile: a 48x32x40 film in FP32x2, three passes of ~10 us a step, 31 ->
 * 24 us; a 64^3 blend in FP64 15.4 -> 14.1 ms an iteration; the launches around
 * the contour loop of a 32x16 film 307 -> 296 us.
 */
#pragma once

#include <cuda_runtime.h>

#include <utility>

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
/* The next kernel's CTAs may start where there is room; late enough that they do not
 * hold an SM for long that another stream could use. */
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... K, typename... A>
inline cudaError_t pdl_launch(void (*kernel)(K...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
