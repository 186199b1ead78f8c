// Chained kernel launches (programmatic dependent launch).
//
// A call of this library is a short chain of kernels (x conversion, SpMV,
// fix-up), and a solver makes one call after another.  Launched with
// `launch_chained`, a kernel may start while the kernel before it on the
// stream drains: its blocks run up to wait_for_previous(), which returns once
// the previous kernel has completed and its writes are visible.  Before that
// call a chained kernel touches nothing but its plan's own read-only arrays
// (task lists, values, columns), which were in place before the plan was
// handed out; x, y and every scratch array come after it.  In every chained
// kernel some warp of the grid waits (a warp with no task may return before),
// so no kernel of a chain completes before its predecessor, and lets its
// successor in at its start (release_next()): the successor's blocks are only
// scheduled once all of its own have started.
// A kernel that is resident early sees x, converted x, chunk sums, carries and
// partial sums change in its lifetime, so it reads them by ld_prev(): the
// read-only path (__ldg, ld.global.nc) and __restrict__ are for the plan's
// arrays alone.  They promise data that nobody writes while the kernel runs,
// and let the compiler move a load across the wait.
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
// A value that an earlier kernel of the chain may have written (after the wait).
// Volatile, so that it stays behind the wait; a plain dereference did too, but
// its schedule took 40 registers in place of 32 in the kernels with a hot-column
// window (R-MAT 2^22 212.6 -> 229.4 us; with these 213).
#define VNEC_LD_PREV(T, OP, REG)                                                        \
  __device__ __forceinline__ T ld_prev(const T* p) {                                    \
    T v;                                                                                \
    asm volatile("ld.global." OP " %0, [%1];" : "=" REG(v) : "l"(p));                   \
    return v;                                                                           \
  }
VNEC_LD_PREV(double, "f64", "d")
VNEC_LD_PREV(float, "f32", "f")
VNEC_LD_PREV(int, "s32", "r")
#undef VNEC_LD_PREV
__device__ __forceinline__ double2 ld_prev(const double2* p) {
  double2 v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 ld_prev(const float2* p) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ int2 ld_prev(const int2* p) {
  int2 v;
  asm volatile("ld.global.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ int4 ld_prev(const int4* p) {
  int4 v;
  asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// The same, read once (streaming).
__device__ __forceinline__ double2 ld_prev_once(const double2* p) {
  double2 v;
  asm volatile("ld.global.cs.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
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
