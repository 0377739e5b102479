// Kernels of the time loop follow each other in one stream (or graph), each
// reading what the one before wrote.  launch_chained lets the next one's blocks
// be scheduled while the last blocks of the one before finish; chain_wait, the
// first thing such a kernel does, holds them until that kernel has ended and its
// writes are visible.  This hides the launch and the block start: smooth 100^2
// 2028 -> 1962 us, learned 512^2 723 -> 670, 4096^2 14.6 -> 13.9 ms.
// chain_release, which lets them be scheduled, stands near a kernel's end, before
// its last stores: at the top, the waiting blocks took their places while every
// block of the one before still held its own, two on one SM and none on another
// (smooth 100^2 2847 us, FP32 257 x 193 920 instead of 709).
// A chained kernel reads state by ordinary or L2 loads and TMA, after the wait;
// never by read-only loads (ld.global.nc), which may see lines cached before it.
#pragma once

#include <cuda_runtime.h>

namespace wenofd {

template <typename... P, typename... A>
cudaError_t launch_chained(void (*fn)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, const A &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

namespace dev {

#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace dev
}  // namespace wenofd
