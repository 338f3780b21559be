// ppm_launch.cuh -- launches of the solve's kernel chain.
//
// A solve is a chain of short kernels on one stream; on a small grid the gaps between them
// (about 2 us each: the next kernel's launch begins when the last block of the one before
// has finished) cost as much as the kernels.  Programmatic dependent launch overlaps them:
// a kernel of the chain is launched while the one before it runs, and waits (pdl_wait)
// before it touches memory until that kernel has completed and its writes are visible.
// Every kernel that launch_chain launches calls pdl_wait first thing and then lets the next
// one start (pdl_next), so a kernel's completion implies that of all before it.  The wait is
// for the kernel just before in the stream alone: behind a caller's kernel that starts its
// dependents early, without having waited itself, it would not order the call after what the
// caller queued before that.  So on a caller's stream the first kernel of a call is launched
// without the attribute (launch_link, chained = false); a context's own stream holds nothing
// but its kernels and copies.  Captured into a graph the order is the same (programmatic
// edges).  Whole step,
// ordinary launches -> chain, with both reconstructions of a small batch in one launch
// (us): 16^3 167 -> 113, 1-D 100 cells 104 -> 81, 256x192 161 -> 128, 37x24x53 244 -> 199,
// 24 patches 608 -> 573.
#pragma once

#include <cuda_runtime.h>

namespace ppm {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_begin() {
  pdl_wait();
  pdl_next();
}

// kernel<<<grid, block, smem, st>>>(args...), as a link of the chain or (chained = false) as
// an ordinary launch
template <class... P, class... A>
inline cudaError_t launch_link(bool chained, void (*kernel)(P...), int64_t grid, int block,
                               size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <class... P, class... A>
inline cudaError_t launch_chain(void (*kernel)(P...), int64_t grid, int block, size_t smem,
                                cudaStream_t st, const A&... args) {
  return launch_link(true, kernel, grid, block, smem, st, args...);
}

}  // namespace ppm
