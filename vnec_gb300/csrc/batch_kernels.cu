// Batched multi-right-hand-side SpMV kernel (batch.h): one persistent launch
// over the task list of the block-diagonal concatenation of the batch.
//
// Lane l of a warp serves right-hand sides [sub * R, sub * R + R) with
// sub = l % L, R = k / L, and slot l / L of the S = 32 / L (value, column)
// slots the warp reads at every step (lanes of a slot read the same pair, a
// broadcast).  A ROWS task holds G = S / V rows, V = 2^vwl slots per row:
// entry j of row g sits at base + (j / V) * S + g * V + j % V, each lane
// gathers R consecutive values of row `column` of X with 16-byte vector loads
// (so the L lanes of a slot read the whole k-wide X row), and the V slots of a
// row are summed with xor-shuffles.  CHUNK tasks (pieces of rows longer than
// the grouping limit) use all S slots for one row; their sums go to chunk_sum
// and the last chunk of a row to arrive (an arrival counter per long row,
// reset by that chunk) adds the row's chunk sums in chunk order, so no second
// kernel is needed.
//
// Arithmetic forms (codecs):
//   FP64 — FP64 values, X and FMA;
//   FP32 — FP32 values, X rounded to FP32 once per call by a preceding kernel,
//          FP32 products and per-lane accumulation; slot, chunk and long-row
//          sums in FP64;
//   DF32 — values stored as FP32 (hi, lo) truncation-split pairs, X split once
//          per call; Dekker products and TwoSum accumulation on the FP32 pipe
//          (FP64-level accuracy), FP64 slot/chunk sums.  When the split kernel
//          flags an X value outside the split range, the same launch computes
//          in FP64 (value = hi + lo, FP64 X).
//
// What bounds it: FP64 from k = 8 on the FP64 pipe (17 M nonzeros, k = 32: 870 us
// of FMAs in a 952 us call), the others the latency and requests of the X gathers.
// So FP64 additions and conversions are kept few (slots are summed by halving the
// right-hand sides a lane holds, FP32 sums are widened by integer operations), and
// the FP32 and double-float loops fetch the next steps' columns and values before
// they wait for X (FP64 loops do not: the registers cost more warps than it hides;
// k = 32 971 -> 997 us).  Measured on lognormal batches of 17 M and, in brackets,
// 0.8 M nonzeros, us a call, against one task per warp, slots summed by a full
// butterfly, no fetch-ahead and half or a quarter of the right-hand sides per lane:
//   k =        2               8               32
//   FP64   187 -> 103      304 -> 264      1063 -> 952   (122 -> 43)
//   FP32   129 -> 74       142 -> 111       410 -> 301   (60 -> 41)
//   DF32   168 -> 91       218 -> 174       643 -> 587   (94 -> 31)

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "batch.h"
#include "common.h"
#include "df32.cuh"
#include "launch.cuh"

namespace vnec {
namespace {

constexpr unsigned kFull = 0xffffffffu;

struct BatchArgs {
  const int4* tasks;
  long long num_tasks;
  const void* val;
  const int32_t* col;
  const int32_t* rowid;
  const int32_t* long_row;
  const int32_t* long_first;
  const int32_t* chunk_long;
  double* chunk_sum;
  int* chunk_count;
  const void* x;       // X in the codec's element type
  const double* x64;   // DF32: the FP64 X (guard path)
  const int* flag;     // DF32: X outside the split range this call
  double* y;
  int klog2;  // k = 1 << klog2
  int llog2;  // lanes per slot L = 1 << llog2
};

// R consecutive elements of type T at p: 32-byte loads (WIDE, p aligned to 32
// bytes: the library's own converted X) or 16-, 8- or 4-byte ones (VEC, p
// aligned to the smaller of 16 bytes and the elements' size), else one by one.
template <bool WIDE, bool VEC, typename T, int R> __device__ __forceinline__ void load_vec(const T* p, T (&v)[R]) {
  constexpr int bytes = R * (int)sizeof(T);
  if constexpr (!VEC) {
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = ld_prev(p + r);
  } else if constexpr (WIDE && bytes >= 32) {
#pragma unroll
    for (int i = 0; i < bytes / 32; ++i) {
      uint32_t w[8];
      asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                   : "l"(reinterpret_cast<const char*>(p) + 32 * i));
      memcpy(reinterpret_cast<char*>(v) + 32 * i, w, 32);
    }
  } else if constexpr (bytes >= 16) {
#pragma unroll
    for (int i = 0; i < bytes / 16; ++i) {
      const int4 q = ld_prev(reinterpret_cast<const int4*>(p) + i);
      memcpy(reinterpret_cast<char*>(v) + 16 * i, &q, 16);
    }
  } else if constexpr (bytes == 8) {
    const int2 q = ld_prev(reinterpret_cast<const int2*>(p));
    memcpy(v, &q, 8);
  } else {
    const int q = ld_prev(reinterpret_cast<const int*>(p));
    memcpy(v, &q, 4);
  }
}

// The first `n` of R values (n a power of two, uniform) to p.
template <bool VEC, int R> __device__ __forceinline__ void store_y(double* p, const double (&v)[R], int n) {
  if constexpr (VEC && R > 1) {
#pragma unroll
    for (int i = 0; i < R / 2; ++i)
      if (2 * i + 1 < n) reinterpret_cast<double2*>(p)[i] = make_double2(v[2 * i], v[2 * i + 1]);
    if (n == 1) p[0] = v[0];
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (i < n) p[i] = v[i];
  }
}

struct CodecF64 {
  static constexpr bool kPairReduce = false, kOwnX = false;
  using V = double;
  using X = double;
  struct A {
    double s;
  };
  __device__ static A zero() { return A{0.0}; }
  __device__ static void mac(A& a, V v, X x) { a.s = fma(v, x, a.s); }
  __device__ static double out(const A& a) { return a.s; }
};

struct CodecF32 {
  static constexpr bool kPairReduce = false, kOwnX = true;
  using V = float;
  using X = float;
  struct A {
    float s;
  };
  __device__ static A zero() { return A{0.f}; }
  __device__ static void mac(A& a, V v, X x) { a.s = fmaf(v, x, a.s); }
  __device__ static double out(const A& a) { return widen(a.s); }
};

// Double-float: value (hi, lo) times x (hi, lo), Dekker product with FMA,
// TwoSum into (s, c).
struct CodecDF32 {
  static constexpr bool kPairReduce = true, kOwnX = true;
  using V = float2;
  using X = float2;
  struct A {
    float s, c;
  };
  // a += the (s, c) pair of the lane `off` away (TwoSum of the high parts).
  __device__ static void add_shfl(A& a, int off) {
    add(a, __shfl_xor_sync(0xffffffffu, a.s, off), __shfl_xor_sync(0xffffffffu, a.c, off));
  }
  // The lane keeps one of a and b (b in the upper lanes), gets that of the
  // other lane and leaves the sum in a.
  __device__ static void fold(A& a, const A& b, bool hi, int off) {
    const A give = hi ? a : b, own = hi ? b : a;
    const A got{__shfl_xor_sync(0xffffffffu, give.s, off), __shfl_xor_sync(0xffffffffu, give.c, off)};
    a = hi ? got : own;  // the lower lane's pair first, whichever lane adds
    add(a, hi ? own.s : got.s, hi ? own.c : got.c);
  }
  __device__ static void add(A& a, float s2, float c2) {
    const float t = __fadd_rn(a.s, s2);
    const float bb = __fsub_rn(t, a.s);
    const float e = __fadd_rn(__fsub_rn(a.s, __fsub_rn(t, bb)), __fsub_rn(s2, bb));
    a.s = t;
    a.c = __fadd_rn(a.c, __fadd_rn(c2, e));
  }
  __device__ static A zero() { return A{0.f, 0.f}; }
  __device__ static void mac(A& a, V v, X x) {
    const DF r = df_mac(DF{a.s, a.c}, v.x, v.y, x.x, x.y);
    a.s = r.s;
    a.c = r.c;
  }
  __device__ static double out(const A& a) { return df_to_f64(DF{a.s, a.c}); }
};

// FP64 from split values and FP64 X: the guard path of DF32 plans.
struct CodecDF32Guard {
  static constexpr bool kPairReduce = false, kOwnX = false;
  using V = float2;
  using X = double;
  struct A {
    double s;
  };
  __device__ static A zero() { return A{0.0}; }
  __device__ static void mac(A& a, V v, X x) {
    a.s = fma(static_cast<double>(v.x) + static_cast<double>(v.y), x, a.s);
  }
  __device__ static double out(const A& a) { return a.s; }
};

__device__ __forceinline__ double shfl_val(double v, int src) { return __shfl_sync(kFull, v, src); }
__device__ __forceinline__ float shfl_val(float v, int src) { return __shfl_sync(kFull, v, src); }
__device__ __forceinline__ float2 shfl_val(float2 v, int src) {
  return make_float2(__shfl_sync(kFull, v.x, src), __shfl_sync(kFull, v.y, src));
}

// STAGED: each task's (column, value) entries are read 32 * kStageRounds at a
// time with one coalesced load per lane per 32 entries, and every step's pair
// reaches its slot's lanes by shuffles, so inside the step loop only the X
// gathers wait on memory.  Otherwise every step's pair is loaded by the slot's
// lanes (broadcast), U steps in flight.
constexpr int kStageRounds = 4;

//
// TL > 0: a warp takes 2^TL consecutive tasks at once, W = 32 >> TL lanes each.
// A layout of L lanes per slot then runs with L >> TL lanes that hold 2^TL times
// the right-hand sides: every slot's sums are those of TL = 0, bit for bit, but
// fewer lanes read each column and value and X comes in wider loads.
template <class Cd, int R, int U, bool STAGED, bool VEC, bool AHEAD, bool HALVE, int TL = 0>
__device__ __forceinline__ void run_tasks(const BatchArgs& a, const typename Cd::X* x) {
  static_assert(TL == 0 || (!STAGED && AHEAD), "several tasks per warp run the fetch-ahead loop");
  using V = typename Cd::V;
  using X = typename Cd::X;
  constexpr int W = 32 >> TL;  // lanes of a task
  const int lane = threadIdx.x & (W - 1);
  const int k = 1 << a.klog2;
  const int S = 32 >> a.llog2;      // slots per step
  const int ll = a.llog2 - TL;      // lanes of a slot
  const int slot = lane >> ll, sub = lane & ((1 << ll) - 1);
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  const V* __restrict__ val = static_cast<const V*>(a.val);
  const X* xs = x + sub * R;
  for (long long w0 = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w0 << TL < a.num_tasks;
       w0 += nw) {
    const long long t = (w0 << TL) + ((threadIdx.x & 31) >> (5 - TL));
    // A warp's last tasks may be missing: no rows, no steps.
    const int4 raw = TL == 0 || t < a.num_tasks ? __ldg(a.tasks + t) : make_int4(0, 0, 0, kSlicedZero);
    const int base = raw.x, row_base = raw.y, kind = raw.w & 15, vwl = (raw.w >> 4) & 15, nrows = raw.w >> 8;
    const int steps = TL > 0 && kind == kSlicedZero ? 0 : raw.z;
    if (kind == kSlicedZero) {
      for (int i = lane; i < (nrows << a.klog2); i += W)
        a.y[((size_t)__ldg(a.rowid + row_base + (i >> a.klog2)) << a.klog2) + (i & (k - 1))] = 0.0;
      if (TL == 0) continue;
    }
    const V* vp = val + base + slot;
    const int32_t* cp = a.col + base + slot;
    typename Cd::A acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = Cd::zero();
    int s = 0;
    if constexpr (STAGED) {
      const int E = steps * S;  // entries of the task
      const int spr = 32 / S;   // steps per 32 entries (= L)
      const int32_t* cb = a.col + base;
      const V* vb = val + base;
      for (int e0 = 0; e0 < E; e0 += 32 * kStageRounds) {
        int creg[kStageRounds];
        V vreg[kStageRounds];
#pragma unroll
        for (int b = 0; b < kStageRounds; ++b) {
          const int e = e0 + b * 32 + lane;
          creg[b] = e < E ? __ldcs(cb + e) : 0;
          vreg[b] = e < E ? __ldcs(vb + e) : V{};
        }
#pragma unroll
        for (int b = 0; b < kStageRounds; ++b) {
          const int sb = (e0 + b * 32) / S;  // first step held by register round b
          if (sb >= steps) break;
          for (int j = 0; j < spr; j += U) {
            int c[U];
            V v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int src = (((j + u) * S) & 31) + slot;
              c[u] = __shfl_sync(kFull, creg[b], src);
              v[u] = shfl_val(vreg[b], src);
            }
            X xv[U][R];
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (j + u < spr && sb + j + u < steps) load_vec<Cd::kOwnX, VEC>(xs + ((size_t)c[u] << a.klog2), xv[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (j + u < spr && sb + j + u < steps)
#pragma unroll
                for (int r = 0; r < R; ++r) Cd::mac(acc[r], v[u], xv[u][r]);
          }
        }
      }
      s = steps;
    }
    if constexpr (AHEAD) {
      // U steps at a time; the next U steps' columns and values are fetched before
      // these steps' X rows are waited for.
      if (s < steps) {
        int c[U];
        V v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (u < steps) {
            c[u] = __ldcs(cp + u * S);
            v[u] = __ldcs(vp + u * S);
          }
        for (; s < steps; s += U) {
          X xv[U][R];
          V w[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (s + u < steps) {
              load_vec<Cd::kOwnX, VEC>(xs + ((size_t)c[u] << a.klog2), xv[u]);
              w[u] = v[u];
            }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (s + U + u < steps) {
              c[u] = __ldcs(cp + (s + U + u) * S);
              v[u] = __ldcs(vp + (s + U + u) * S);
            }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (s + u < steps)
#pragma unroll
              for (int r = 0; r < R; ++r) Cd::mac(acc[r], w[u], xv[u][r]);
        }
      }
    } else {
      for (; s + U <= steps; s += U) {
        int c[U];
        V v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          c[u] = __ldcs(cp + (s + u) * S);
          v[u] = __ldcs(vp + (s + u) * S);
        }
        X xv[U][R];
#pragma unroll
        for (int u = 0; u < U; ++u) load_vec<Cd::kOwnX, VEC>(xs + ((size_t)c[u] << a.klog2), xv[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int r = 0; r < R; ++r) Cd::mac(acc[r], v[u], xv[u][r]);
      }
      for (; s < steps; ++s) {
        const int c = __ldcs(cp + s * S);
        const V v = __ldcs(vp + s * S);
        X xv[R];
        load_vec<Cd::kOwnX, VEC>(xs + ((size_t)c << a.klog2), xv);
#pragma unroll
        for (int r = 0; r < R; ++r) Cd::mac(acc[r], v, xv[r]);
      }
    }
    // Slots to sum: the whole warp for a chunk, the V slots of a row otherwise.
    // At each level the two halves of the lanes split the right-hand sides they
    // still hold, so R values over n slots take R - 1 or fewer additions per lane
    // instead of R log2(n); every sum is the butterfly's.
    const int span = kind == kSlicedZero ? 0 : kind == kSlicedChunk ? W : 1 << (ll + vwl);
    double d[R];
    int width = R, at = 0;  // this lane ends with right-hand sides [at, at + width) of its R
    bool writes = true;
    if constexpr (!HALVE) {
#pragma unroll
      for (int r = 0; r < R; ++r) d[r] = Cd::out(acc[r]);
      for (int off = 1 << ll; off < span; off <<= 1)
#pragma unroll
        for (int r = 0; r < R; ++r) d[r] += __shfl_xor_sync(kFull, d[r], off);
      writes = kind == kSlicedChunk ? slot == 0 : (slot & ((1 << vwl) - 1)) == 0;
    } else if constexpr (Cd::kPairReduce) {
      // Double-float: sum the slots as (hi, lo) pairs on the FP32 pipe and
      // convert once (each FP64 operation costs 64 FP32 issue slots here).
#pragma unroll
      for (int lev = 0; lev < 5; ++lev) {
        const int off = 1 << (ll + lev);
        if (off >= span) break;
        const bool hi = (lane & off) != 0;
        if ((R >> lev) > 1) {
#pragma unroll
          for (int j = 0; j < (R >> lev) / 2; ++j) Cd::fold(acc[j], acc[j + (R >> lev) / 2], hi, off);
          width >>= 1;
          at += hi ? width : 0;
        } else {
          Cd::add_shfl(acc[0], off);
          writes = writes && !hi;
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (r < width) d[r] = Cd::out(acc[r]);
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) d[r] = Cd::out(acc[r]);
#pragma unroll
      for (int lev = 0; lev < 5; ++lev) {
        const int off = 1 << (ll + lev);
        const bool adds = off < span;  // the same for all lanes of a task
        if (TL == 0 ? !adds : !__any_sync(kFull, adds)) break;
        const bool hi = (lane & off) != 0;
        if ((R >> lev) > 1) {
#pragma unroll
          for (int j = 0; j < (R >> lev) / 2; ++j) {
            const double keep = hi ? d[j + (R >> lev) / 2] : d[j], give = hi ? d[j] : d[j + (R >> lev) / 2];
            const double sum = keep + __shfl_xor_sync(kFull, give, off);
            if (adds) d[j] = sum;
          }
          if (adds) {
            width >>= 1;
            at += hi ? width : 0;
          }
        } else {
          const double sum = d[0] + __shfl_xor_sync(kFull, d[0], off);
          if (adds) {
            d[0] = sum;
            writes = writes && !hi;
          }
        }
      }
    }
    if (TL == 0 ? kind == kSlicedChunk : __any_sync(kFull, kind == kSlicedChunk)) {
      const bool chunk = kind == kSlicedChunk;
      if (chunk && writes) store_y<VEC>(a.chunk_sum + ((size_t)row_base << a.klog2) + sub * R + at, d, width);
      __threadfence();
      __syncwarp();
      int li = 0, c0 = 0, c1 = 0, last = 0;
      if (chunk) {
        li = __ldg(a.chunk_long + row_base);
        c0 = __ldg(a.long_first + li);
        c1 = __ldg(a.long_first + li + 1);
        if (lane == 0) last = atomicAdd(a.chunk_count + li, 1) == c1 - c0 - 1;
      }
      last = __shfl_sync(kFull, last, 0, W);
      if (last) {
        __threadfence();
        const size_t yrow = (size_t)__ldg(a.long_row + li) << a.klog2;
        for (int j = lane; j < k; j += W) {
          double sum = 0.0;
          for (int c = c0; c < c1; ++c) sum += __ldcg(a.chunk_sum + ((size_t)c << a.klog2) + j);
          a.y[yrow + j] = sum;
        }
        if (lane == 0) a.chunk_count[li] = 0;
      }
    }
    if (kind == kSlicedRows) {
      const int g = slot >> vwl;
      if (writes && g < nrows)
        store_y<VEC>(a.y + ((size_t)__ldg(a.rowid + row_base + g) << a.klog2) + sub * R + at, d, width);
    }
  }
}

template <class Cd, int R, int U, bool STAGED, bool VEC, bool AHEAD, bool HALVE, int TL, int B>
__global__ void __launch_bounds__(256, B) batch_kernel(const BatchArgs a) {
  release_next();
  wait_for_previous();
  run_tasks<Cd, R, U, STAGED, VEC, AHEAD, HALVE, TL>(a, static_cast<const typename Cd::X*>(a.x));
}

// UG: the guard's steps in flight; its loop neither stages nor fetches ahead, so
// that it does not raise the kernel's registers.
template <int R, int U, int UG, bool STAGED, bool VEC, bool AHEAD>
__global__ void __launch_bounds__(256) batch_df32_kernel(const BatchArgs a) {
  release_next();
  wait_for_previous();
  if (*reinterpret_cast<const volatile int*>(a.flag))
    run_tasks<CodecDF32Guard, R, UG, false, VEC, false, true>(a, a.x64);
  else
    run_tasks<CodecDF32, R, U, STAGED, VEC, AHEAD, true>(a, static_cast<const float2*>(a.x));
}

// Steps in flight per lane: 8 / R (at least 2), doubled in mode 1; mode 2 stages
// the entries in registers with the mode-0 step count.  The fetch-ahead loops (modes
// 0 and 1 of FP32 and DF32) hold the next steps' columns and values too, and the
// double-float pairs are twice as wide, so there the full count costs more warps
// than it hides: 112 to 238 registers where these take 64 to 128.  Explicit layouts
// of 14 M nonzeros and, in brackets, 0.8 M, time against the loop without
// fetch-ahead at mode 1's full count (geometric means over k and chunk lengths):
//   DF32   R = 1: 16 steps 1.74 (0.63), 8 0.96 (0.46), 6 0.74 (0.43), 5 0.66 (0.44), 4 0.68 (0.44);
//          staged 8 against 4: 1.78 (1.80)
//          R = 2:  8 steps 0.97 (0.47), 6 0.95 (0.45), 4 0.79 (0.45), 3 0.71 (0.45)
//          R = 4:  4 steps 0.89 (0.48), 3 0.77 (0.49), 2 0.76 (0.53)
//          R = 8:  4 steps 1.10 (0.48), 3 0.79 (0.46), 2 0.83 (0.46)
//   FP32   R = 1: 16 steps 1.15 (0.59), 12 1.08 (0.58), 8 0.96 (0.72), 6 0.80 (0.62), 4 0.81 (0.76)
//          R = 2:  8 steps 1.06 (0.81), 6 0.82 (0.68), 5 0.84 (0.71), 4 0.85 (0.69)
//          R = 4:  4 steps 0.77 (0.62), 3 0.73 (0.57), 2 0.79 (0.63)
//          R = 8:  4 steps 0.78 (0.48), 3 0.69 (0.54), 2 0.68 (0.58)
constexpr int steps_in_flight(int precision, int R, int mode) {
  if (precision == kPrecDF32) {
    if (R == 1) return mode == 1 ? 5 : 4;
    if (mode == 1 || (mode == 0 && R != 4)) return 3;
  }
  if (precision == kPrecFP32) {
    if (mode == 1 && R == 4) return 3;
    if ((mode == 1 && R <= 2) || (mode == 0 && R == 1)) return 6;
  }
  return (R >= 4 ? 2 : 8 / R) * (mode == 1 ? 2 : 1);
}

using BatchKernel = void (*)(BatchArgs);
template <int R, int MODE, bool VEC> BatchKernel kernel_for(int precision) {
  constexpr bool ST = MODE == 2, AHEAD = !ST;
  switch (precision) {
    case kPrecFP32:
      return &batch_kernel<CodecF32, R, steps_in_flight(kPrecFP32, R, MODE), ST, VEC, AHEAD, true, 0,
                           ST && R == 1 ? 4 : 0>;  // 64 registers, not 80: 14 M nonzeros 1.13x, 0.8 M 1.01x
    case kPrecDF32:
      return &batch_df32_kernel<R, steps_in_flight(kPrecDF32, R, MODE), steps_in_flight(kPrecFP64, R, 0), ST, VEC, AHEAD>;
    default:
      // R of 1 and 2 with twice the steps: the plain butterfly leaves the compiler
      // a better schedule (1.06 to 1.5x over k and sizes; R = 4, 8: 0.9x).
      return &batch_kernel<CodecF64, R, steps_in_flight(kPrecFP64, R, MODE), ST, VEC, false, !(MODE == 1 && R <= 2), 0, 0>;
  }
}

template <int R, bool VEC = true> BatchKernel kernel_for_mode(int precision, int mode) {
  return mode == 2   ? kernel_for<R, 2, VEC>(precision)
         : mode == 1 ? kernel_for<R, 1, VEC>(precision)
                     : kernel_for<R, 0, VEC>(precision);
}

// Several FP32 tasks per warp (BatchMatrix::tasks_log2), by the right-hand sides
// per lane: 8 with two tasks, 4 with four (k = 4), 2 with two (k = 2).
BatchKernel pick_shared(int r, int tasks_log2, bool vec) {
  if (r == 8 && tasks_log2 == 1) return &batch_kernel<CodecF32, 8, steps_in_flight(kPrecFP32, 8, 0), false, true, true, true, 1, 0>;
  if (r == 4 && tasks_log2 == 2)
    return vec ? &batch_kernel<CodecF32, 4, steps_in_flight(kPrecFP32, 4, 0), false, true, true, true, 2, 0>
               : &batch_kernel<CodecF32, 4, steps_in_flight(kPrecFP32, 4, 0), false, false, true, true, 2, 0>;
  if (r == 2 && tasks_log2 == 1)
    return vec ? &batch_kernel<CodecF32, 2, steps_in_flight(kPrecFP32, 2, 0), false, true, true, true, 1, 0>
               : &batch_kernel<CodecF32, 2, steps_in_flight(kPrecFP32, 2, 0), false, false, true, true, 1, 0>;
  return nullptr;
}

// `vec`: X and Y are 16-byte aligned.  Layouts of 2 and 4 right-hand sides per
// lane also run without (plans whose layout the caller did not fix).
BatchKernel pick_kernel(int precision, int r, int mode, bool vec = true) {
  switch (r) {
    case 1: return kernel_for_mode<1>(precision, mode);
    case 2: return vec ? kernel_for_mode<2>(precision, mode) : kernel_for_mode<2, false>(precision, mode);
    case 4: return vec ? kernel_for_mode<4>(precision, mode) : kernel_for_mode<4, false>(precision, mode);
    case 8: return vec ? kernel_for_mode<8>(precision, mode) : nullptr;
    default: return nullptr;
  }
}

int log2i(int v) {
  int l = 0;
  while ((1 << l) < v) ++l;
  return l;
}

}  // namespace

int batch_grid(int precision, int rhs_per_lane, int warps_per_block, int mode) {
  const BatchKernel fn = pick_kernel(precision, rhs_per_lane, mode);
  if (!fn || (warps_per_block != 4 && warps_per_block != 8)) return 0;
  int dev = 0, sms = 0, per_sm = 0;
  if (!VNEC_CUDA(cudaGetDevice(&dev)) ||
      !VNEC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) ||
      !VNEC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, warps_per_block * 32, 0)))
    return 0;
  return sms * std::max(per_sm, 1);
}

bool batch_spmm(const BatchMatrix& m, const double* X, double* Y, cudaStream_t s) {
  return batch_spmm_range(m, X, Y, s, 0, m.num_tasks, 0, m.n_cols, true);
}

bool batch_spmm_range(const BatchMatrix& m, const double* X, double* Y, cudaStream_t s, int64_t t0, int64_t t1,
                      int64_t c0, int64_t c1, bool first) {
  if (!batch_supported(m.k, m.lanes)) {
    set_error("batch: unsupported k / lanes");
    return false;
  }
  const int R = (m.k / m.lanes) << m.tasks_log2;
  const void* xin = X;
  const long long off = (long long)c0 * m.k, nx = (long long)(c1 - c0) * m.k;
  if (m.precision == kPrecFP32) {
    if (nx > 0 && !round_to_f32(X + off, static_cast<float*>(m.xbuf) + off, nx, s)) return false;
    xin = m.xbuf;
  } else if (m.precision == kPrecDF32) {
    if (first && !VNEC_CUDA(cudaMemsetAsync(m.flag, 0, sizeof(int), s))) return false;
    if (nx > 0 && !split_to_df32(X + off, static_cast<float2*>(m.xbuf) + off, nx, m.flag, s)) return false;
    xin = m.xbuf;
  }
  if (t1 <= t0) return true;
  BatchArgs a;
  a.tasks = reinterpret_cast<const int4*>(m.tasks) + t0;
  a.num_tasks = t1 - t0;
  a.val = m.val;
  a.col = m.col;
  a.rowid = m.rowid;
  a.long_row = m.long_row;
  a.long_first = m.long_first;
  a.chunk_long = m.chunk_long;
  a.chunk_sum = m.chunk_sum;
  a.chunk_count = m.chunk_count;
  a.x = xin;
  a.x64 = X;
  a.flag = m.flag;
  a.y = Y;
  a.klog2 = log2i(m.k);
  a.llog2 = log2i(m.lanes);
  const bool vec = ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Y)) & 15) == 0;
  const BatchKernel fn =
      m.tasks_log2 > 0 ? pick_shared(R, m.tasks_log2, vec) : pick_kernel(m.precision, R, m.mode, vec || R == 1);
  if (!fn) {
    set_error("batch: x and y must be 16-byte aligned for this plan's layout");
    return false;
  }
  // Persistent warps stride the task list; with per_task every warp takes one
  // task and the hardware dispatches the blocks in task order, so the tasks in
  // flight stay a compact window of the list (and of X's rows).
  const long long per_block = (long long)m.warps_per_block << m.tasks_log2;
  const long long per_task_grid = (a.num_tasks + per_block - 1) / per_block;
  if (m.per_task && per_task_grid > 0x7fffffffLL) {
    set_error("batch: too many tasks for one launch with one warp per task");
    return false;
  }
  const int grid = m.per_task ? (int)per_task_grid
                              : (int)std::min<long long>(m.grid, std::max<long long>(1, (a.num_tasks + 7) / 8));
  return launch_chained(fn, (unsigned)grid, (unsigned)(m.warps_per_block * 32), 0, s, a);
}

}  // namespace vnec
