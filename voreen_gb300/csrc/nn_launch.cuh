// Launches of the learned form's kernels one after another on a stream, the
// next one's CTAs resident and past their index arithmetic when the last CTA
// of the one before ends (programmatic dependent launch). The 14 kernels of a
// 960x540 frame's upsampler 454 -> 437 us, the three convolutions of a training
// step's 64 -> 64 layer on 8x96x96 78 -> 71.
#pragma once
#include <cuda_runtime.h>

namespace {

// First touch of anything in global memory comes after this: it returns when
// every kernel before this one has completed and its writes are visible. What
// such a kernel may have written is not read by ld.global.nc (no __ldg, no
// const __restrict__), which promises that nothing is written while the grid
// lives. Each kernel waits here, so a kernel that starts early has all but its
// predecessor behind it.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute chained{};
    chained.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    chained.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    // a graph's nodes are launched ahead anyhow, and its programmatic edges cost
    // more than they give (the upsampler's graph 438 us without, 444 with)
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const bool known = cudaStreamIsCapturing(s, &capture) == cudaSuccess;
    if (!known) cudaGetLastError();
    c.attrs = &chained;
    c.numAttrs = known && capture == cudaStreamCaptureStatusNone ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...), last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}

}  // namespace
