// Chained kernel launches (programmatic dependent launch).
//
// A call of this library is a short chain of kernels (x conversion, SpMV,
// fix-up), and a solver makes one call after another.  Launched with
// `launch_chained`, a kernel may start while the kernel before it on the
// stream drains: its blocks run up to wait_for_previous(), which returns once
// the previous kernel has completed and its writes are visible.  Before that
// call a chained kernel touches nothing but its plan's own read-only arrays
// (task lists, values, columns), which were in place before the plan was
// handed out; x, y and every scratch array come after it.  Every chained
// kernel waits on every path, so completion is transitive along the chain,
// and lets its successor in at its start (release_next()): the successor's
// blocks are only scheduled once all of its own have started.
// After a kernel that does not release (a caller's), a copy, a memset or an
// event wait, a chained launch is an ordinary stream-ordered one.
//
// What bounds small calls without it is the drain of one grid and the start of
// the next, 1.5 to 3 us a launch.  Measured back to back on GB300 (us a call):
// uniform 65,536 x 16 FP64 8.4 -> 6.5, its FP32 form 12.4 -> 7.9, DF32 22.9 ->
// 14.0; R-MAT 2^13 FP64 10.6 -> 7.3; R-MAT 2^22 FP64 (three launches) 215 -> 208;
// 70 shapes and forms from 10^5 to 10^7 nonzeros: 1.32x in the geometric mean.
// Loading a task's first columns and values before the wait as well gains up to
// 10% more on small grids but costs the stencils 7% and R-MAT 2^22 5%.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "common.h"

namespace vnec {

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

template <typename... P, typename... A>
bool launch_chained(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return VNEC_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...));
}

}  // namespace vnec
