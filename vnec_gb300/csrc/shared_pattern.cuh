// Shared-pattern tasks (kSlicedShared, sliced.h): step k's column in every row is
// the row's first column plus one offset for the whole task.
//
// The warp turns the task's stored gaps into offsets (a prefix sum over the
// lanes) and leaves them in shared memory, where one 16-byte read, the same
// address in every lane, gives four steps' offsets.  A row's x pointer moves to
// its first column once, so a step costs a value load, an x load with one
// multiply-add for its address, and the FMA.  (With a shuffle per step and
// predicated steps throughout, the FP32 form took 25 instructions a step, and
// instruction issue, 64% busy, and not memory held it back.)  27-point stencil,
// us a call: FP32 form 160^3 114.6 -> 98.3, BF16 100^3 26.0 -> 24.2; FP32 type,
// whose kernel walked 2-byte gaps per entry before, 100^3 35.1 -> 22.4; FP64
// 100^3 58.4 -> 52.6, 144^3 146 -> 143 (126 of them FP64 FMAs).
#pragma once

#include <cstdint>

namespace vnec {

constexpr int kPatternSteps = 32;  // a shared-pattern task has at most this many steps

// `buf`: kPatternSteps ints of this warp, 16-byte aligned.
__device__ __forceinline__ const int4* pattern_offsets(const uint16_t* pat, int steps, int lane, int* buf) {
  int off = lane < steps ? __ldg(pat + lane) : 0;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, off, o);
    if (lane >= o) off += t;
  }
  buf[lane] = off;
  __syncwarp();
  return reinterpret_cast<const int4*>(buf);
}

// Offsets of steps k .. k + N - 1; k and N are multiples of 4.
template <int N> __device__ __forceinline__ void pattern_at(const int4* offs, int k, int (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N / 4; ++i) {
    const int4 q = offs[k / 4 + i];
    o[4 * i] = q.x;
    o[4 * i + 1] = q.y;
    o[4 * i + 2] = q.z;
    o[4 * i + 3] = q.w;
  }
}

}  // namespace vnec
