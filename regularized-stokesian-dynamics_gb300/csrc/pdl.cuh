// Programmatic dependent launch.  A step of a small system is a chain of short
// kernels, and most of its time the gaps between them (2.2 us each in one
// stream).  A kernel launched with pdl_launch is set up while the one before
// it in its stream still runs, and waits for that one's end and memory in
// pdl_enter, before it touches anything.  pdl_enter also lets the next such
// kernel be set up, one ahead and no more, so that waiting CTAs never fill the
// GPU.  Every kernel launched so has to begin with it (each kernel's end then
// implies the end of all before it in the stream).
#pragma once
#include "rsd_internal.cuh"

namespace {

__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
void pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
  RSD_LAUNCH_NOTE();
}

}  // namespace
