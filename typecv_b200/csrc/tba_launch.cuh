// Launches of a solve's kernels, each before the kernel ahead of it in the stream has ended.
//
// An iteration of the explicit system is ten short kernels, each of which needs all of the one before.
// Launched the ordinary way a kernel's blocks are set up once the last block of the kernel before is gone,
// about 2 us of an idle device per kernel.  Launched with launch_dependent they are set up as soon as the
// kernel before has started all of its own, take room that it leaves free, and wait in after_previous() for
// its end and its writes: six iterations on a 7-camera window 880 -> 770 us.  (The batch's
// kernels are nodes of a graph, where it gained nothing: 24 windows 3.35 ms either way.)
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace tba {

// First statement of every kernel that launch_dependent launches: the kernels before have ended and their
// writes are visible; the next kernel's blocks may then be set up.  (A kernel that skipped the wait would
// let the next one start before the kernel ahead of both has ended.)  Launched the ordinary way, nothing.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t s,
                                    A... args) {
  cudaLaunchAttribute early{};
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &early;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace tba
