// Launches with programmatic stream serialization: a kernel may be scheduled while the one before it in the stream drains.
//
// Contract of every kernel launched through launch_pdl():
//   * every thread executes pdl_wait() before it touches global memory (and before it returns): until then the kernels
//     before it may still be running.  Barriers, tensor memory and tensor-map prefetches are set up ahead of it;
//   * pdl_trigger() comes after pdl_wait() and after the CTA's tensor-memory allocation: it lets the next kernel's CTAs
//     take the places that this kernel's CTAs leave.  All CTAs of this kernel are running or done by then, so none of them
//     can be kept out, and the next kernel's allocation cannot get in front of this one's.
// Kernels that wait for other CTAs or other GPUs use neither: they start after, and are followed by, complete kernels.
// What it gives is the set-up and scheduling time of a launch, 1 - 1.5 us of the 2 - 3 us that a small kernel takes.  A trigger
// costs about 0.5 ns per CTA, one CTA of the whole chip after the other, which only large grids of short CTAs notice: an
// embedding lookup of 32768 CTAs of 1.5 KB takes 34.6 us with it and 18.4 us without, RMSNorm of 65536 x 256 (16384 CTAs of
// 4 KB) 17.6 and 11.8, but LayerNorm of 30000 x 768 (7500 CTAs of 12 KB) 15.8 and 16.4.  pdl_trigger_work() leaves the trigger
// of such grids to the end of the kernel.
#pragma once
#include <cuda_runtime.h>

namespace ftk {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// `cta_bytes`: what a CTA reads and writes
__device__ __forceinline__ void pdl_trigger_work(int cta_bytes) {
  if (gridDim.x <= 2048 || cta_bytes >= 8192) pdl_trigger();
}

template <typename... P, typename... A>
static inline int launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace ftk
