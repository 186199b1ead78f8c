// Sliced row-group SpMV (VNEC-S counterpart, src/operation/src/spmv_vnec_S_for_mxv.c:589-660).
//
// One warp per task (sliced.h).  For a ROWS task of vector width VW the warp
// reads `steps` rows of 32 consecutive entries — 256 B of FP64 values and
// 128 B of columns per step, fully coalesced — so lane l accumulates entries
// of group row l / VW; a VW-lane xor-shuffle reduction finishes each row
// (VW = 1: the reference's cross-row kernel, one lane per row, no reduction).
// CHUNK tasks do the same for 32-wide pieces of long rows and a second launch
// adds the pieces of each long row in chunk order.  Values and columns are
// read once (no L1 allocation, L2 evict-first policy); x is gathered by
// ordinary loads (launch.cuh).
// FP64 work: one FMA per entry plus log2(VW) adds per row.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.h"
#include "launch.cuh"
#include "long_rows.cuh"
#include "prefetch.cuh"
#include "shared_pattern.cuh"
#include "sliced.h"

namespace vnec {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarpsPerBlock = 8;

// Loads with explicit cache policies (hint 1): values and columns are read
// once — no L1 allocation, L2 policy evict_first — while x is kept (L1
// evict_last, L2 policy evict_last) so its hot part stays cached across tasks.
struct Policies {
  unsigned long long once, keep;
};
__device__ __forceinline__ Policies make_policies() {
  Policies p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p.once));
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p.keep));
  return p;
}
__device__ __forceinline__ double ld_once(const double* p, unsigned long long pol) {
  double v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_once(const float* p, unsigned long long pol) {
  float v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ int ld_once(const int* p, unsigned long long pol) {
  int v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ double ld_keep(const double* p, unsigned long long pol) {
  double v;
  asm volatile("ld.global.L1::evict_last.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_keep(const float* p, unsigned long long pol) {
  float v;
  asm volatile("ld.global.L1::evict_last.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}

// Streamed value/column loads with no L1 allocation and no L2 policy.
__device__ __forceinline__ double ld_na(const double* p) {
  double v;
  asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_na(const float* p) {
  float v;
  asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ int ld_na(const int* p) {
  int v;
  asm("ld.global.nc.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ double ld_l1_keep(const double* p) {
  double v;
  asm volatile("ld.global.L1::evict_last.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_l1_keep(const float* p) {
  float v;
  asm volatile("ld.global.L1::evict_last.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

// Cache-hint variants H: 0 streaming (.cs) loads of values/columns and
// plain x gathers; 1 explicit L1/L2 policies; 2 values/columns without L1
// allocation; 3 as 2 with x gathers marked L1 evict-last.
template <int H, typename T> __device__ __forceinline__ T ld_stream_h(const T* p, const Policies& pol) {
  if constexpr (H == 0) return __ldcs(p);
  else if constexpr (H == 1) return ld_once(p, pol.once);
  else return ld_na(p);
}
template <int H, typename T> __device__ __forceinline__ T ld_x_h(const T* p, const Policies& pol) {
  if constexpr (H == 0 || H == 2) return ld_prev(p);
  else if constexpr (H == 1) return ld_keep(p, pol.keep);
  else return ld_l1_keep(p);
}


template <typename V> __device__ __forceinline__ V fmav(V a, V b, V c);
template <> __device__ __forceinline__ double fmav<double>(double a, double b, double c) { return fma(a, b, c); }
template <> __device__ __forceinline__ float fmav<float>(float a, float b, float c) { return fmaf(a, b, c); }

// Dense-block entries (VNEC-D counterpart): 4 consecutive values starting at
// column c; x is read at c..c+3 (guarded by n_cols).
template <typename V> struct Quad;
template <> struct Quad<double> {
  __device__ static void load(const double* p, double (&v)[4]) {
    const double2 a = __ldcs(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
};
template <> struct Quad<float> {
  __device__ static void load(const float* p, float (&v)[4]) {
    const float4 a = __ldcs(reinterpret_cast<const float4*>(p));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  }
};

// One warp per task, U blocks of a lane in flight, the last round predicated instead
// of taking its blocks one by one.  What bounds it: latency (a block's columns, then
// its x), and for FP64 the FP64 pipe on filled-up blocks.  So what is loaded ahead is
// weighed against the warps its registers cost, by the longest task of the plan:
//   kDenseColumns: the columns of a round, values with each block's x (32 registers)
//   kDenseValues:  a round's columns and values together (30 to 38)
//   kDenseNext:    these, and the next round's columns (38 to 64)
// us, one block after the other with four columns loaded -> kDenseColumns (U = 4, FP32
// 6), kDenseValues (U = 2), kDenseNext (U = 2):
//   FP64  2 random columns a row   35.1 -> 31.1, 40.8, 32.6   band of 6, 3 M rows  49.8 -> 43.5, 44.7, 49.7
//         5                        31.0 -> 30.8, 41.7, 30.2   band of 16           12.4 -> 12.5, 10.7, 8.9
//         9                        32.9 -> 33.2, 39.1, 33.0   blocks of 4          18.5 -> 13.5, 15.5, 17.6
//         7                        29.2 -> 36.6, 37.2, 28.3   blocks of 32         16.6 -> 19.9, 16.6, 14.2
//   FP32  7 random columns a row   24.7 -> 24.2, 26.5, 21.5   band of 6, 3 M rows  41.1 -> 27.1, 21.8, 27.2
//         3                        26.8 -> 21.9, 23.6, 22.5   blocks of 24         10.3 -> 5.8, 5.2, 5.6
//         8                        24.7 -> 25.1, 26.9, 21.5   blocks of 32         8.3 -> 7.2, 6.1, 5.3
// With tasks of more than 10 blocks a lane, where a chain of rounds ends the call, U =
// 2 loses: lognormal rows FP64 108 (U = 4) against 121, FP32 81 (6) against 89; 16
// random columns a row, FP64, 49 against 61.  Nor do the next columns pay there: 12
// random columns a row, FP32, 87 (kDenseValues, 6) against 106, lognormal 18 against 24.
enum DenseLoads : int { kDenseColumns, kDenseValues, kDenseNext };
constexpr int kDenseShort = 10;
// Up to here kDenseNext; FP32 plans of 9 and 10 blocks keep kDenseValues (27-point
// stencil 65^3 10.5 us against 12.3, 160^3 112 against 115; 9 random columns 24 and 23).
template <typename V> constexpr int kDenseNextMost = sizeof(V) == 8 ? 10 : 8;
template <typename V> constexpr int kDenseAhead = sizeof(V) == 8 ? 4 : 6;
template <typename V> constexpr int kDenseFew = sizeof(V) == 8 ? 3 : 6;
template <typename V> constexpr DenseLoads kDenseFewLoads = sizeof(V) == 8 ? kDenseColumns : kDenseValues;
template <typename V> constexpr int kDenseFewAhead = sizeof(V) == 8 ? 4 : 2;

template <typename V, int U, DenseLoads LOADS>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
dense_block_kernel(const SlicedTask* __restrict__ tasks, long long num_tasks, const V* __restrict__ val,
                   const int32_t* __restrict__ col, const int32_t* __restrict__ rowid, const V* x, int n_cols, V* y, V* chunk_sum) {
  const long long w = ((long long)blockIdx.x * kWarpsPerBlock) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  release_next();
  if (w >= num_tasks) return;
  const int4 raw = __ldg(reinterpret_cast<const int4*>(tasks) + w);
  const int base = raw.x, row_base = raw.y, steps = raw.z, meta = raw.w;
  const int kind = meta & 15, vwl = (meta >> 4) & 15, nrows = (meta >> 8) & 0xff;
  wait_for_previous();
  if (kind == kSlicedZero) {
    if (lane < nrows) y[rowid[row_base + lane]] = V(0);
    return;
  }
  const V* vp = val + (size_t)(base + lane) * 4;
  const int32_t* cp = col + base + lane;
  V acc = V(0);
  int next[U];
  if constexpr (LOADS == kDenseNext) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < steps) next[u] = __ldcs(cp + u * 32);
  }
  for (int k = 0; k < steps; k += U) {
    int c[U];
    V v[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u < steps) {
        c[u] = LOADS == kDenseNext ? next[u] : __ldcs(cp + (k + u) * 32);
        if constexpr (LOADS != kDenseColumns) Quad<V>::load(vp + (size_t)(k + u) * 128, v[u]);
      }
    if constexpr (LOADS == kDenseNext) {
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (k + U + u < steps) next[u] = __ldcs(cp + (k + U + u) * 32);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u < steps) {
        V xv[4];
        if constexpr (LOADS == kDenseColumns) Quad<V>::load(vp + (size_t)(k + u) * 128, v[u]);
#pragma unroll
        for (int l = 0; l < 4; ++l) xv[l] = c[u] + l < n_cols ? ld_prev(x + c[u] + l) : V(0);
#pragma unroll
        for (int l = 0; l < 4; ++l) acc = fmav<V>(v[u][l], xv[l], acc);
      }
  }
  for (int off = (1 << vwl) >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(kFull, acc, off);
  if (kind == kSlicedChunk) {
    if (lane == 0) chunk_sum[row_base] = acc;
  } else {
    const int g = lane >> vwl;
    if ((lane & ((1 << vwl) - 1)) == 0 && g < nrows) y[rowid[row_base + g]] = acc;
  }
}

// Address of x for a (possibly hot-relabelled) column.
template <bool HOT, typename V>
__device__ __forceinline__ const V* x_at(const V* x, const V* xh, int ncols, int c) {
  if constexpr (HOT) return c < ncols ? x + c : xh + (c - ncols);
  else return x + c;
}

// Output of row `row`: the sum, or alpha * sum + beta * z[row] + gamma.
// z is not restrict-qualified: it may alias y (the thread reads z[row] before
// it writes y[row], and no other thread touches that entry).
template <bool EPI, typename V>
__device__ __forceinline__ V epi_out(V acc, int row, const SlicedEpilogue& ep) {
  if constexpr (EPI) {
    const double g = ep.gamma_dev ? fma(ep.gamma_dev_scale, *ep.gamma_dev, ep.gamma) : ep.gamma;
    double r = fma(ep.alpha, static_cast<double>(acc), g);
    if (ep.z) r = fma(ep.beta, static_cast<double>(static_cast<const V*>(ep.z)[row]), r);
    return static_cast<V>(r);
  } else {
    return acc;
  }
}

// One warp task (the body of sliced_kernel and of the DF32 guard kernel).
// SH: the plan has shared-pattern tasks; plans without them run the SH = false
// build, whose registers that path does not raise.
template <typename V, int U, int H, bool HOT, bool EPI, bool SH = false>
__device__ __forceinline__ void sliced_task(long long w, int lane, const SlicedTask* __restrict__ tasks,
                                            const V* __restrict__ val, const int32_t* __restrict__ col,
                                            const int32_t* __restrict__ rowid, const V* x, V* y, V* chunk_sum,
                                            const V* xh, int ncols,
                                            const SlicedEpilogue& ep, const uint16_t* __restrict__ col16,
                                            const int32_t* __restrict__ first,
                                            const SlicedPrefetch& pf = SlicedPrefetch(),
                                            const uint16_t* __restrict__ pat16 = nullptr, int* s_off = nullptr) {
  const int4 raw = __ldg(reinterpret_cast<const int4*>(tasks) + w);
  const int base = raw.x, row_base = raw.y, steps = raw.z, meta = raw.w;
  const int kind = meta & 15, vwl = (meta >> 4) & 15, nrows = (meta >> 8) & 0xff;
  // The entries and task metadata ahead of this task, into L2 (prefetch.cuh).
  if (pf.entries > 0) {
    prefetch_l2_task_meta(pf, w, base, row_base, kind != kSlicedChunk, tasks, first, rowid, SH ? pat16 : nullptr, lane);
    const long long e0 = base + pf.entries, len = 32LL * steps;
    if (kind != kSlicedZero && e0 + len <= pf.n_entries) {
      prefetch_l2_range(val + e0, len, lane);
      if (SH && (meta & kSlicedShared)) {
      } else if (meta & kSlicedDelta)
        prefetch_l2_range(col16 + e0, len, lane);
      else
        prefetch_l2_range(col + e0, len, lane);
    }
  }
  wait_for_previous();
  if (kind == kSlicedZero) {
    if (lane < nrows) {
      const int row = rowid[row_base + lane];
      y[row] = epi_out<EPI>(V(0), row, ep);
    }
    return;
  }
  if (SH && (meta & kSlicedShared)) {
    // One row per lane, all with the same column gaps (shared_pattern.cuh).
    const int4* offs = pattern_offsets(pat16 + (base >> 5), steps, lane, s_off);
    const V* xr = x + (lane < nrows ? __ldg(first + row_base + lane) : 0);
    const V* vp = val + base + lane;
    V acc = V(0);
    int k = 0;
    for (; k + U <= steps; k += U) {
      V v[U], xv[U];
      int o[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = __ldcs(vp + (k + u) * 32);
      pattern_at<U>(offs, k, o);
#pragma unroll
      for (int u = 0; u < U; ++u) xv[u] = ld_prev(xr + o[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) acc = fmav<V>(v[u], xv[u], acc);
    }
    for (; k < steps; k += 4) {
      V v[4], xv[4];
      int o[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u < steps) v[u] = __ldcs(vp + (k + u) * 32);
      pattern_at<4>(offs, k, o);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u < steps) xv[u] = ld_prev(xr + o[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (k + u < steps) acc = fmav<V>(v[u], xv[u], acc);
    }
    if (lane < nrows) {
      const int row = rowid[row_base + lane];
      y[row] = epi_out<EPI>(acc, row, ep);
    }
    return;
  }
  if (meta & kSlicedDelta) {
    // One row per lane, columns as 16-bit deltas from the row's first column.
    const V* vp = val + base + lane;
    const uint16_t* dp = col16 + base + lane;
    int c = lane < nrows ? __ldg(first + row_base + lane) : 0;
    V acc = V(0);
    int k = 0;
    for (; k + U <= steps; k += U) {
      int cc[U];
      V v[U], xv[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        cc[u] = __ldcs(dp + (k + u) * 32);
        v[u] = __ldcs(vp + (k + u) * 32);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        c += cc[u];
        cc[u] = c;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) xv[u] = ld_prev(x_at<HOT>(x, xh, ncols, cc[u]));
#pragma unroll
      for (int u = 0; u < U; ++u) acc = fmav<V>(v[u], xv[u], acc);
    }
    for (; k < steps; ++k) {
      c += __ldcs(dp + k * 32);
      acc = fmav<V>(__ldcs(vp + k * 32), ld_prev(x_at<HOT>(x, xh, ncols, c)), acc);
    }
    if (lane < nrows) {
      const int row = rowid[row_base + lane];
      y[row] = epi_out<EPI>(acc, row, ep);
    }
    return;
  }
  const V* vp = val + base + lane;
  const int32_t* cp = col + base + lane;
  Policies pol{0, 0};
  if constexpr (H == 1) pol = make_policies();
  V acc = V(0);
  int k = 0;
  for (; k + U <= steps; k += U) {
    int c[U];
    V v[U], xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      c[u] = ld_stream_h<H>(cp + (k + u) * 32, pol);
      v[u] = ld_stream_h<H>(vp + (k + u) * 32, pol);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) xv[u] = ld_x_h<H>(x_at<HOT>(x, xh, ncols, c[u]), pol);
#pragma unroll
    for (int u = 0; u < U; ++u) acc = fmav<V>(v[u], xv[u], acc);
  }
  for (; k < steps; ++k)
    acc = fmav<V>(ld_stream_h<H>(vp + k * 32, pol),
                  ld_x_h<H>(x_at<HOT>(x, xh, ncols, ld_stream_h<H>(cp + k * 32, pol)), pol), acc);
  for (int off = (1 << vwl) >> 1; off > 0; off >>= 1) acc += __shfl_xor_sync(kFull, acc, off);
  if (kind == kSlicedChunk) {
    if (lane == 0) chunk_sum[row_base] = acc;
  } else {
    const int g = lane >> vwl;
    if ((lane & ((1 << vwl) - 1)) == 0 && g < nrows) {
      const int row = rowid[row_base + g];
      y[row] = epi_out<EPI>(acc, row, ep);
    }
  }
}

template <typename V, int U, int H, bool HOT = false, bool EPI = false, bool SH = false>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
sliced_kernel(const SlicedTask* __restrict__ tasks, long long num_tasks, const V* __restrict__ val,
              const int32_t* __restrict__ col, const int32_t* __restrict__ rowid, const V* x, V* y, V* chunk_sum,
              const V* xh = nullptr, int ncols = 0,
              SlicedEpilogue ep = SlicedEpilogue(), const uint16_t* __restrict__ col16 = nullptr,
              const int32_t* __restrict__ first = nullptr, SlicedPrefetch pf = SlicedPrefetch(),
              const uint16_t* __restrict__ pat16 = nullptr) {
  __shared__ __align__(16) int s_off[SH ? kWarpsPerBlock : 1][kPatternSteps];
  const long long w = ((long long)blockIdx.x * kWarpsPerBlock) + (threadIdx.x >> 5);
  release_next();
  if (w >= num_tasks) return;
  sliced_task<V, U, H, HOT, EPI, SH>(w, threadIdx.x & 31, tasks, val, col, rowid, x, y, chunk_sum, xh, ncols, ep,
                                     col16, first, pf, pat16, s_off[SH ? threadIdx.x >> 5 : 0]);
}

// FP64 recompute of a DF32 call whose x left the split range: a small grid of
// warps striding the task list, so that the launch costs next to nothing in
// the usual case (flag clear: every block returns at once).  The last block to
// finish clears the flag, guard[0], for the next call; guard[1] counts them.
template <bool HOT>
__global__ void __launch_bounds__(kWarpsPerBlock * 32)
sliced_guard_kernel(int* guard, const SlicedTask* __restrict__ tasks, long long num_tasks,
                    const double* __restrict__ val, const int32_t* __restrict__ col,
                    const int32_t* __restrict__ rowid, const double* x, double* y, double* chunk_sum,
                    const double* xh, int ncols,
                    const uint16_t* __restrict__ col16, const int32_t* __restrict__ first) {
  release_next();
  wait_for_previous();
  if (*reinterpret_cast<const volatile int*>(guard) == 0) return;
  const SlicedEpilogue ep;
  const long long stride = (long long)gridDim.x * kWarpsPerBlock;
  for (long long w = (long long)blockIdx.x * kWarpsPerBlock + (threadIdx.x >> 5); w < num_tasks; w += stride)
    sliced_task<double, 8, 0, HOT, false>(w, threadIdx.x & 31, tasks, val, col, rowid, x, y, chunk_sum, xh, ncols,
                                          ep, col16, first);
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(guard + 1, 1) == (int)gridDim.x - 1) {
    atomicExch(guard + 1, 0);
    atomicExch(guard, 0);
  }
}

template <typename V, bool EPI = false>
__global__ void sliced_long_fixup(const int32_t* __restrict__ long_row, const int32_t* __restrict__ long_first,
                                  const int32_t* __restrict__ long_heavy, long long num_long, long long num_heavy,
                                  long long heavy_sub, unsigned light_blocks, const V* chunk_sum, V* y,
                                  SlicedEpilogue ep = SlicedEpilogue()) {
  release_next();
  wait_for_previous();
  long_rows_fixup<V>(long_first, long_heavy, num_long, num_heavy, heavy_sub, light_blocks, chunk_sum,
                     [&](long long i, V s) {
                       const int row = long_row[i];
                       y[row] = epi_out<EPI>(s, row, ep);
                     });
}

template <typename V>
__global__ void epilogue_kernel(V* y, long long n, SlicedEpilogue ep) {
  release_next();
  wait_for_previous();
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double g = ep.gamma_dev ? fma(ep.gamma_dev_scale, *ep.gamma_dev, ep.gamma) : ep.gamma;
    double r = fma(ep.alpha, static_cast<double>(y[i]), g);
    if (ep.z) r = fma(ep.beta, static_cast<double>(static_cast<const V*>(ep.z)[i]), r);
    y[i] = static_cast<V>(r);
  }
}

template <typename V>
bool launch_dense(const SlicedMatrix& m, const void* x, void* y, cudaStream_t s) {
  const long long grid = (m.num_tasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
  if (grid > 0x7fffffffLL) {
    set_error("dense blocks: too many tasks for one launch");
    return false;
  }
  const auto kern = m.longest <= kDenseFew<V> ? dense_block_kernel<V, kDenseFewAhead<V>, kDenseFewLoads<V>>
                    : m.longest <= kDenseNextMost<V> ? dense_block_kernel<V, 2, kDenseNext>
                    : m.longest <= kDenseShort ? dense_block_kernel<V, 2, kDenseValues>
                                               : dense_block_kernel<V, kDenseAhead<V>, kDenseValues>;
  return launch_chained(kern, (unsigned)grid, kWarpsPerBlock * 32, 0, s, m.tasks, m.num_tasks,
                        static_cast<const V*>(m.val), m.col, m.rowid, static_cast<const V*>(x), (int)m.n_cols,
                        static_cast<V*>(y), static_cast<V*>(m.chunk_sum));
}

template <typename V>
__global__ void gather_hot(const V* x, const int32_t* __restrict__ hot_cols, int n, V* xh) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  release_next();
  const int c = i < n ? __ldg(hot_cols + i) : 0;
  wait_for_previous();
  if (i < n) xh[i] = ld_prev(x + c);
}

template <typename V>
bool launch_gather_hot(const SlicedMatrix& m, const void* x, cudaStream_t s) {
  return launch_chained(gather_hot<V>, (unsigned)((m.hot + 255) / 256), 256, 0, s, static_cast<const V*>(x),
                        m.hot_cols, m.hot, static_cast<V*>(m.xhot));
}

template <typename V, int U, int H, bool HOT, bool EPI = false, bool SH = false>
bool launch_main(const SlicedMatrix& m, const void* x, void* y, cudaStream_t s,
                 const SlicedEpilogue& ep = SlicedEpilogue()) {
  auto kern = sliced_kernel<V, U, H, HOT, EPI, SH>;
  // No shared memory (SH: 1 KB a block): give the unified L1/shared array to L1.
  static std::atomic<unsigned long long> configured{0};  // per instantiation, per device
  if (!once_per_device(configured, [&] {
        return VNEC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, SH ? 12 : 0));
      }))
    return false;
  const long long grid = (m.num_tasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
  if (grid > 0x7fffffffLL) {
    set_error("sliced: too many tasks for one launch");
    return false;
  }
  if (HOT && !m.hot_ready && !launch_gather_hot<V>(m, x, s)) return false;
  return launch_chained(kern, (unsigned)grid, kWarpsPerBlock * 32, 0, s, m.tasks, m.num_tasks,
                        static_cast<const V*>(m.val), m.col, m.rowid, static_cast<const V*>(x), static_cast<V*>(y),
                        static_cast<V*>(m.chunk_sum), static_cast<const V*>(m.xhot), (int)m.n_cols, ep, m.col16,
                        m.first, m.pf, m.pat16);
}

template <typename V, int U, bool HOT>
bool launch_hints(const SlicedMatrix& m, const void* x, void* y, cudaStream_t s) {
  // Shared-pattern tasks need 16-bit deltas, which a hot-column window rules out.
  if constexpr (!HOT)
    if (m.pat16 && m.cache_hints == 0) return launch_main<V, U, 0, false, false, true>(m, x, y, s);
  switch (m.cache_hints) {
    case 1: return launch_main<V, U, 1, HOT>(m, x, y, s);
    case 2: return launch_main<V, U, 2, HOT>(m, x, y, s);
    case 3: return launch_main<V, U, 3, HOT>(m, x, y, s);
    default: return launch_main<V, U, 0, HOT>(m, x, y, s);
  }
}

template <typename V, bool HOT>
bool launch_unroll(const SlicedMatrix& m, const void* x, void* y, cudaStream_t s) {
  switch (m.unroll) {
    case 4: return launch_hints<V, 4, HOT>(m, x, y, s);
    case 12: return launch_hints<V, 12, HOT>(m, x, y, s);
    case 16: return launch_hints<V, 16, HOT>(m, x, y, s);
    default: return launch_hints<V, 8, HOT>(m, x, y, s);
  }
}

template <typename V, bool HOT>
bool launch_fused(const SlicedMatrix& m, const void* x, void* y, cudaStream_t s, const SlicedEpilogue& ep) {
  if constexpr (!HOT)
    if (m.pat16) switch (m.unroll) {
        case 4: return launch_main<V, 4, 0, false, true, true>(m, x, y, s, ep);
        case 8: return launch_main<V, 8, 0, false, true, true>(m, x, y, s, ep);
        case 16: return launch_main<V, 16, 0, false, true, true>(m, x, y, s, ep);
        default: return launch_main<V, 12, 0, false, true, true>(m, x, y, s, ep);
      }
  switch (m.unroll) {
    case 4: return launch_main<V, 4, 0, HOT, true>(m, x, y, s, ep);
    case 8: return launch_main<V, 8, 0, HOT, true>(m, x, y, s, ep);
    case 16: return launch_main<V, 16, 0, HOT, true>(m, x, y, s, ep);
    default: return launch_main<V, 12, 0, HOT, true>(m, x, y, s, ep);
  }
}

template <typename V>
bool launch_variant(const SlicedMatrix& m, const void* x, void* y, cudaStream_t s) {
  return m.hot > 0 ? launch_unroll<V, true>(m, x, y, s) : launch_unroll<V, false>(m, x, y, s);
}

template <typename V>
bool launch(const SlicedMatrix& m, const void* x, void* y, cudaStream_t s, cudaEvent_t* ev,
            const SlicedEpilogue* epi) {
  if (ev && !VNEC_CUDA(cudaEventRecord(ev[0], s))) return false;
  // The fused epilogue runs at the plan's unroll with default cache hints;
  // dense-block plans apply it as a separate pass.
  const bool fused = epi && m.vpe == 1;
  if (m.num_tasks > 0) {
    bool ok;
    if (m.vpe == 4)
      ok = launch_dense<V>(m, x, y, s);
    else if (fused)
      ok = m.hot > 0 ? launch_fused<V, true>(m, x, y, s, *epi) : launch_fused<V, false>(m, x, y, s, *epi);
    else
      ok = launch_variant<V>(m, x, y, s);
    if (!ok) return false;
  }
  if (ev && !VNEC_CUDA(cudaEventRecord(ev[1], s))) return false;
  if (m.num_long > 0) {
    const int b = 128;
    const FixupGrid g = fixup_grid(m, b);
    auto kern = fused ? sliced_long_fixup<V, true> : sliced_long_fixup<V, false>;
    if (!launch_chained(kern, g.total, b, 0, s, m.long_row, m.long_first, m.long_heavy, (long long)m.num_long,
                        (long long)m.num_heavy, (long long)m.heavy_sub, g.light, static_cast<const V*>(m.chunk_sum),
                        static_cast<V*>(y), fused ? *epi : SlicedEpilogue()))
      return false;
  }
  if (epi && !fused && !apply_epilogue(y, m.n_rows, sizeof(V) == 8, *epi, s)) return false;
  if (ev && !VNEC_CUDA(cudaEventRecord(ev[2], s))) return false;
  return true;
}

}  // namespace

bool sliced_guard_f64(const SlicedMatrix& m, const double* x, double* y, int* flag, cudaStream_t s) {
  // The guard only runs for DF32 plans, whose FP64 values sit in m.val and
  // whose hot columns (if any) are served from x directly through hot_cols.
  int dev = 0, sms = 0;
  if (!VNEC_CUDA(cudaGetDevice(&dev)) || !VNEC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)))
    return false;
  const long long need = (m.num_tasks + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(need, 8LL * sms));
  if (m.hot > 0) {
    if (!launch_gather_hot<double>(m, x, s)) return false;
    return launch_chained(sliced_guard_kernel<true>, grid, kWarpsPerBlock * 32, 0, s, flag, m.tasks, m.num_tasks,
                          static_cast<const double*>(m.val), m.col, m.rowid, x, y, static_cast<double*>(m.chunk_sum),
                          static_cast<const double*>(m.xhot), (int)m.n_cols, m.col16, m.first);
  }
  return launch_chained(sliced_guard_kernel<false>, grid, kWarpsPerBlock * 32, 0, s, flag, m.tasks, m.num_tasks,
                        static_cast<const double*>(m.val), m.col, m.rowid, x, y, static_cast<double*>(m.chunk_sum),
                        nullptr, 0, m.col16, m.first);
}

bool sliced_spmv(const SlicedMatrix& m, bool fp64, const void* x, void* y, cudaStream_t s, cudaEvent_t* ev,
                 const SlicedEpilogue* epi) {
  return fp64 ? launch<double>(m, x, y, s, ev, epi) : launch<float>(m, x, y, s, ev, epi);
}

bool sliced_gather_hot(const SlicedMatrix& m, bool fp64, const void* x, cudaStream_t s) {
  if (m.hot <= 0) return true;
  return fp64 ? launch_gather_hot<double>(m, x, s) : launch_gather_hot<float>(m, x, s);
}

bool apply_epilogue(void* y, long long n, bool fp64, const SlicedEpilogue& e, cudaStream_t s) {
  if (n <= 0) return true;
  const int tb = 256;
  const unsigned grid = (unsigned)std::min<long long>((n + tb - 1) / tb, 152LL * 16);
  return fp64 ? launch_chained(epilogue_kernel<double>, grid, tb, 0, s, static_cast<double*>(y), n, e)
              : launch_chained(epilogue_kernel<float>, grid, tb, 0, s, static_cast<float*>(y), n, e);
}

}  // namespace vnec
