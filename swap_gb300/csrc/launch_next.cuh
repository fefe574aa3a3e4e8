// launch_next.cuh -- kernels of one stream that start while the one before
// them drains (programmatic dependent launch).
//
// A step of a middle-sized grid is a chain of some fifty short kernels, and
// between two of them the GPU empties and fills again: about 2 us each.  A
// kernel launched by launch_next may start as soon as every block of the
// kernel before it in the stream has started; it calls after_previous() before
// it touches memory, which returns when that kernel has ended and its stores
// are visible.  (Its pointers are not __restrict__: a load through one that is
// may be a load of constant memory to the compiler, free to move up past the
// wait.)  What comes after such a kernel by a plain launch, a copy or an
// event waits for its end as always.
//
// Measured, 20 steps: FP32 form 64x64x64 cells 12.2 -> 9.9 ms, 128x64x64 18.4
// -> 16.4, 16x8x12 (the moments' kernels around the passes) 3.62 -> 3.24; FP64
// form 128x64x64 2% less.  Not for the particle passes and the sort's kernels:
// their many blocks, let in early, hold the places that the other stream's
// kernels need (256x128x128 cells 266 -> 322 ms).
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace swapk {

// First in a kernel launched by launch_next (without effect in others): lets
// the next kernel's blocks in, and waits for the kernel before this one.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
cudaError_t launch_next_smem(void (*kernel)(P...), dim3 grid, dim3 block, std::size_t smem, cudaStream_t st, A... a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(a)...);
}
template <class... P, class... A>
cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A... a) {
  return launch_next_smem(kernel, grid, block, 0, st, a...);
}

}  // namespace swapk
