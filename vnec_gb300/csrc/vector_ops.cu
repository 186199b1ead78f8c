// Device reductions for chains of SpMV calls that stay on the GPU (power
// iterations: a dangling-mass dot product, an L1 convergence distance).  Two
// launches with a summation order fixed by n and the vectors' alignment, so the
// result has the same bits on every run: up to SPB_VNEC_DOT_BLOCKS blocks write
// partial sums, one block adds them in block order.
//
// Bound by latency at these sizes (2^20 values are 16.8 MB, 2.5 us at HBM rate):
// a thread has eight values of each vector in flight as 16-byte loads, into four
// sums, and a short vector takes fewer blocks.  One value at a time and always
// 1,024 blocks before: 16,384 values 7.2 -> 4.8 us, 2^20 10.0 -> 8.9 (differences
// 12.6 -> 11.4); long vectors run at HBM rate as before (5 10^7: 124 us, products;
// differences 238 -> 210, two FP64 instructions a value).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.h"
#include "launch.cuh"
#include "vnec_gb300.h"

namespace vnec {
namespace {

constexpr int kDotTpb = 256;

__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
  return s;
}

constexpr int kDotPairs = 4;  // pairs of values in flight per thread
constexpr long long kDotBlockValues = (long long)kDotTpb * 2 * kDotPairs;

// MODE 0: products; 1: absolute differences (compiled apart: chosen at run time,
// both were computed, three FP64 instructions a value).  `vec`: both vectors are
// 16-byte aligned.
template <int MODE>
__global__ void __launch_bounds__(kDotTpb)
dot_partial_kernel(long long n, const double* a, const double* b, bool vec, double* partial) {
  __shared__ double sh[kDotTpb / 32];
  release_next();
  wait_for_previous();
  auto add = [](double acc, double u, double v) {
    if constexpr (MODE == 0)
      return fma(u, v, acc);
    else
      return acc + fabs(u - v);
  };
  double acc[kDotPairs] = {};
  const long long t = (long long)blockIdx.x * kDotTpb + threadIdx.x, stride = (long long)gridDim.x * kDotTpb;
  const long long n2 = vec ? n / 2 : 0;
  const double2 *a2 = reinterpret_cast<const double2*>(a), *b2 = reinterpret_cast<const double2*>(b);
  long long q = t;
  for (; q + (kDotPairs - 1) * stride < n2; q += kDotPairs * stride) {
    double2 u[kDotPairs], v[kDotPairs];
#pragma unroll
    for (int j = 0; j < kDotPairs; ++j) {
      u[j] = ld_prev(a2 + q + j * stride);
      v[j] = ld_prev(b2 + q + j * stride);
    }
#pragma unroll
    for (int j = 0; j < kDotPairs; ++j) acc[j] = add(add(acc[j], u[j].x, v[j].x), u[j].y, v[j].y);
  }
  for (; q < n2; q += stride) {
    const double2 u = ld_prev(a2 + q), v = ld_prev(b2 + q);
    acc[0] = add(add(acc[0], u.x, v.x), u.y, v.y);
  }
#pragma unroll 4
  for (long long i = 2 * n2 + t; i < n; i += stride) acc[0] = add(acc[0], ld_prev(a + i), ld_prev(b + i));
  const double s = block_sum((acc[0] + acc[1]) + (acc[2] + acc[3]), sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kDotTpb)
dot_final_kernel(const double* partial, int n, double* out) {
  __shared__ double sh[kDotTpb / 32];
  release_next();
  wait_for_previous();
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < SPB_VNEC_DOT_BLOCKS / kDotTpb; ++j) {
    const int i = threadIdx.x + j * kDotTpb;
    acc += i < n ? partial[i] : 0.0;
  }
  const double s = block_sum(acc, sh);
  if (threadIdx.x == 0) out[0] = s;
}

}  // namespace
}  // namespace vnec

extern "C" SpB_Info SpB_VNEC_dot_ext(int64_t n, const double* d_a, const double* d_b, int mode, double* d_partial,
                                     double* d_out, void* stream) {
  using namespace vnec;
  clear_error();
  if (n < 0 || (mode != 0 && mode != 1) || !d_partial || !d_out || (n > 0 && (!d_a || !d_b))) {
    set_error("SpB_VNEC_dot_ext: invalid arguments");
    return SpB_FAILURE;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool vec = ((reinterpret_cast<uintptr_t>(d_a) | reinterpret_cast<uintptr_t>(d_b)) & 15) == 0;
  const int blocks =
      (int)std::min<long long>(SPB_VNEC_DOT_BLOCKS, std::max<long long>(1, (n + kDotBlockValues - 1) / kDotBlockValues));
  return launch_chained(mode == 0 ? dot_partial_kernel<0> : dot_partial_kernel<1>, (unsigned)blocks, kDotTpb, 0, s,
                        (long long)n, d_a, d_b, vec, d_partial) &&
                 launch_chained(dot_final_kernel, 1, kDotTpb, 0, s, d_partial, blocks, d_out)
             ? SpB_SUCCESS
             : SpB_FAILURE;
}
