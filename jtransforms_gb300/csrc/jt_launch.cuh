// jt_launch.cuh -- launches that overlap the previous kernel's end
// (programmatic dependent launch).
//
// Short transforms are chains of kernels of a few microseconds, and a launch
// in stream order starts only when the kernel before it has drained.  These
// kernels are launched with programmatic stream serialisation: their blocks
// may be placed as soon as all blocks of the kernel before have begun, and wait
// (pdl_begin, the first thing each thread does) until it has finished and its
// memory is visible, before they touch global memory.  Every thread of such a
// kernel makes that wait, so a chain of them keeps stream order.  Measured
// (GB300, both directions): FloatFFT_2D(2048^2).realForward, six kernels, 64.5 ->
// 55.2 us; DoubleFFT_1D(4096) x 256, two kernels, 43.2 -> 40.0 us.
#pragma once

#include <cuda_runtime.h>

namespace jt {

__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Elementwise kernels, one number a thread: a block lives about as long as those
// two instructions take, so grids above four waves (of 152 SMs, eight blocks of
// 256 each) launch in plain stream order and skip them (FloatFFT_1D(188779) x 64,
// pre/mul/post around a power of two, both directions: 1541 us with them in every
// block, 1411 without).
#define JT_PDL_BLOCKS (4 * 8 * 152)
__device__ __forceinline__ void pdl_begin_few() {
    if (gridDim.x <= JT_PDL_BLOCKS) pdl_begin();
}

// overlap: 0 launches in plain stream order.
template <typename... P, typename... A>
inline cudaError_t pdl_launch_if(bool overlap, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...a) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(a)...);
}
template <typename... P, typename... A>
inline cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&...a) {
    return pdl_launch_if(true, kernel, grid, block, smem, s, static_cast<A &&>(a)...);
}

}  // namespace jt
