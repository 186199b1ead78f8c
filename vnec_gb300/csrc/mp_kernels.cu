// Merge-path CSR SpMV for sm_103a — the GPU counterpart of VNEC-L
// (src/operation/src/spmv_vnec_L_for_mxv.c:124-165) and of its partitioner
// MergePathDivide (src/operation/src/spmv_vnec_common.c:3-33).
//
// Work decomposition.  The merge of the row-end list (row_ptr[1..n]) and the
// nonzero counting list (0..nnz-1) has n_rows + nnz items.  It is cut into
// tiles of a fixed number of items, one CTA per tile; the tile boundaries are
// found once per matrix (plan time) by mp_partition_kernel, so a tile holds a
// bounded number of rows and of nonzeros whatever the row lengths.  Inside a
// tile:
//   1. every thread owns 8 consecutive nonzeros, cut at multiples of 8 of the
//      nonzero index: columns and values come in with 32-byte vector loads
//      (read once, no L1 allocation) straight into registers, and the 8
//      gathers of x are in flight together;
//   2. the tile's row ends are read once, coalesced, and each row with a
//      nonzero in the tile writes its number to a 16-bit slot at its last
//      nonzero's place; a row with none is stored as zero right away.  A
//      thread then finds the row ends among its 8 nonzeros with one 16-byte
//      shared-memory read: no search and no merge walk, and the only FP64
//      work per nonzero is its FMA (an FP64 operation takes the pipe of a
//      whole warp for 16 cycles here, whichever lanes need it);
//   3. carry: a thread whose first row end closes a row that began in an
//      earlier thread adds the partial sums (tails) of the threads in between.
//      Where no row of the tile passes over more than two whole threads, every
//      thread walks back over them.  Else one warp takes all the tile's tails:
//      a lane sums those of four threads, a segmented scan joins the lanes, and
//      the lane goes over its four again to write their rows.  Either way the
//      carries take some 8 to 12 FP64 instructions of a warp next to the 32 of
//      the FMAs.  The tile's own carry-out (partial of its last row) goes to a
//      per-tile scratch slot;
//   4. fix-up (second, tiny launch): rows spanning tiles receive the ordered
//      sum of the carries of the tiles that stopped inside them — the
//      counterpart of the reference's serial carry loop (:159-164).
//
// What bounds it: the x gathers' L1/L2 requests on power-law columns, as in
// the sliced kernel, without its hot-column window, and the FP64 pipe on the
// others: no one unit is full, the phases of a tile do not overlap all the way.
// Measured on GB300 (us a call, FP64 / the FP32 type): R-MAT 2^22, 49 M nonzeros,
// 242 / 175; 27-point stencil 120^3 153 / 76; a million rows of 16, 75 / 63; 20,001
// rows of 1,000, 74 / 42.  Against the pipelined DF32 tiles, whose shared-memory
// merge walk bound them: R-MAT 874, stencil 455.
// Carries: with every row of a warp walked by a lane, and rows past four
// threads shared by the lanes, they took as many FP64 instructions as half the
// nonzeros (28 a tile; FP64 pipe 62% busy): R-MAT 267 / 178, rows of 1,000 101 /
// 47, rows of 16 79 / 64, stencil 155 / 81.  The one warp alone loses on short
// rows (rows of 16: 84, of 4: 105 against 88 with the walk).  Walks over at most 1, 2,
// 3 whole threads: stencil 156, 153, 164; rows of 16 79, 77, 77.
// Tiles: small CTAs overlap the phases best: 128 x 7 items (one thread per 8
// places) against 256 x 7 are 7 to 20% faster, 16 nonzeros a thread up to 15%
// slower on power-law rows.  The default tile of 1,016 items gives all of 128
// threads their 8 places (64 threads, 504 items: 8% slower on R-MAT; 96, 760: 1%
// faster there, 4% slower on the stencil).

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>

#include "common.h"
#include "launch.cuh"
#include "vnec_gb300.h"

namespace vnec {
namespace {

template <typename T> __device__ __forceinline__ T ld_stream(const T* p) { return __ldcs(p); }

template <typename V> __device__ __forceinline__ V fma_v(V a, V b, V c);
template <> __device__ __forceinline__ double fma_v<double>(double a, double b, double c) { return fma(a, b, c); }
template <> __device__ __forceinline__ float fma_v<float>(float a, float b, float c) { return fmaf(a, b, c); }

// Diagonal search of one merge-path boundary (MergePathDivide semantics:
// move right while row_end[pivot] <= diag - pivot - 1).
template <typename Off>
__device__ __forceinline__ Off merge_search(const Off* row_end, Off diag, Off n_rows, Off nnz) {
  Off lo = diag - nnz > 0 ? diag - nnz : 0;
  Off hi = diag < n_rows ? diag : n_rows;
  while (lo < hi) {
    Off p = (lo + hi) >> 1;
    if (row_end[p] <= diag - p - 1)
      lo = p + 1;
    else
      hi = p;
  }
  return lo;
}

template <typename Off>
__global__ void mp_partition_kernel(const Off* __restrict__ row_end, Off n_rows, Off nnz, long long ipc,
                                    long long num_tiles, Off* __restrict__ tile_row, Off* __restrict__ tile_nz) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t > num_tiles) return;
  Off total = n_rows + nnz;
  long long d64 = t * ipc;
  Off diag = d64 < (long long)total ? (Off)d64 : total;
  Off r = merge_search<Off>(row_end, diag, n_rows, nnz);
  tile_row[t] = r;
  tile_nz[t] = diag - r;
}

// N (a multiple of 8) consecutive items as 32-byte vectors; `p` is aligned to
// 32 bytes.
template <int N> __device__ __forceinline__ void load_items(const double* p, double (&v)[N]) {
#pragma unroll
  for (int h = 0; h < N; h += 4)
    asm("ld.global.nc.L1::no_allocate.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(v[h]), "=d"(v[h + 1]), "=d"(v[h + 2]), "=d"(v[h + 3])
        : "l"(p + h));
}
template <int N> __device__ __forceinline__ void load_items(const float* p, float (&v)[N]) {
#pragma unroll
  for (int h = 0; h < N; h += 8)
    asm("ld.global.nc.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[h]), "=f"(v[h + 1]), "=f"(v[h + 2]), "=f"(v[h + 3]), "=f"(v[h + 4]), "=f"(v[h + 5]),
          "=f"(v[h + 6]), "=f"(v[h + 7])
        : "l"(p + h));
}
template <int N> __device__ __forceinline__ void load_items(const int32_t* p, int32_t (&v)[N]) {
#pragma unroll
  for (int h = 0; h < N; h += 8)
    asm("ld.global.nc.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[h]), "=r"(v[h + 1]), "=r"(v[h + 2]), "=r"(v[h + 3]), "=r"(v[h + 4]), "=r"(v[h + 5]),
          "=r"(v[h + 6]), "=r"(v[h + 7])
        : "l"(p + h));
}

constexpr unsigned kNoRow = 0xffffu;  // slot of a nonzero that ends no row
constexpr int E = kMpPlaces;          // nonzeros per thread

// Threads of a tile of `items` merge items: E nonzeros each, and one thread
// more because the tile's first nonzero may lie inside its thread's E.
constexpr int tile_threads(int items) { return ((items + E - 1) / E + 1 + 31) / 32 * 32; }
constexpr int kMaxTileThreads = tile_threads(256 * 10);

constexpr int kReach = 2;  // whole threads without a row end that a walk back crosses at most
constexpr int kRake = 4;   // warps of the default tile: threads whose carries one lane takes

// kRake consecutive shared-memory values as vector loads.
__device__ __forceinline__ void rake_load(const double* p, double (&v)[kRake]) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
}
__device__ __forceinline__ void rake_load(const float* p, float (&v)[kRake]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
}
__device__ __forceinline__ void rake_load(const unsigned short* p, unsigned short (&v)[kRake]) {
  const ushort4 a = *reinterpret_cast<const ushort4*>(p);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
}

// Sum over the lanes back to the nearest one with `ends` (its own value alone
// where that is the lane itself).
template <typename V> __device__ __forceinline__ V rake_scan(V sum, bool ends, int lane) {
  constexpr unsigned kFull = 0xffffffffu;
  const unsigned below = __ballot_sync(kFull, ends) & (kFull >> (31 - lane));
  const int reach = below ? __clz(below) - (31 - lane) : lane;
  const int longest = (int)__reduce_max_sync(kFull, (unsigned)reach);
  for (int d = 1; d <= longest; d <<= 1) {
    const V up = __shfl_up_sync(kFull, sum, d);
    sum += d <= reach ? up : V(0);
  }
  return sum;
}

// One CTA per tile, of at most T threads with E nonzeros each; at least B CTAs
// fit an SM.  Dynamic shared memory: a 16-bit slot per nonzero place, then each
// thread's tail and head sums and the row of its first row end.  `vec`: col and
// val are 32-byte aligned.
template <typename V, typename Off, int T, int B>
__global__ void __launch_bounds__(T, B)
mp_spmv_kernel(const Off* __restrict__ row_end, const int32_t* __restrict__ col, const V* __restrict__ val,
               const V* x, V* y, const Off* __restrict__ tile_row, const Off* __restrict__ tile_nz, Off nnz, bool vec,
               Off* carry_row, V* carry_val) {
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ uint4 s_slots[];
  V* const s_tail = reinterpret_cast<V*>(s_slots + (E / 8) * blockDim.x);
  V* const s_head = s_tail + blockDim.x;
  unsigned short* const s_first = reinterpret_cast<unsigned short*>(s_head + blockDim.x);
  const int tile = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31;
  release_next();
  const Off x0 = tile_row[tile], y0 = tile_nz[tile];
  const int nrows = (int)(tile_row[tile + 1] - x0);
  const int lead = (int)(y0 & (E - 1));   // places before the tile's first nonzero
  const int end = lead + (int)(tile_nz[tile + 1] - y0);  // one past its last
  const Off origin = y0 - lead;           // nonzero at place 0, a multiple of E
  const int q = E * tid;                  // this thread's first place

  // 1. columns and values, then x.  Places outside the tile hold value and x 0.
  V v[E], xv[E];
  {
    const int32_t* cp = col + origin + q;
    const V* vp = val + origin + q;
    int32_t c[E];
    if (vec && q < end && nnz - origin >= q + E) {
      load_items<E>(cp, c);
      load_items<E>(vp, v);
    } else {
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const bool in = q + j >= lead && q + j < end;
        c[j] = in ? ld_stream(cp + j) : 0;
        v[j] = in ? ld_stream(vp + j) : V(0);
      }
    }
    wait_for_previous();
#pragma unroll
    for (int j = 0; j < E; ++j) {
      const bool in = q + j >= lead && q + j < end;
      xv[j] = in ? ld_prev(x + c[j]) : V(0);
      if (!in) v[j] = V(0);
    }
  }

  // 2. row ends: row r of the tile ends after the nonzero at place e - 1; its
  // first nonzero in the tile is at the end of the row before it.
#pragma unroll
  for (int h = 0; h < E / 8; ++h) s_slots[(E / 8) * tid + h] = make_uint4(~0u, ~0u, ~0u, ~0u);
  __syncthreads();
  {
    unsigned short* slot = reinterpret_cast<unsigned short*>(s_slots);
    for (int r = tid; r < nrows; r += blockDim.x) {
      const Off e = row_end[x0 + r], b = r ? row_end[x0 + r - 1] : y0;
      if (e > b)
        slot[(int)(e - y0) + lead - 1] = (unsigned short)r;
      else
        y[x0 + r] = V(0);
    }
  }
  __syncthreads();
  unsigned sw[E / 2];
#pragma unroll
  for (int h = 0; h < E / 8; ++h) {
    const uint4 s4 = s_slots[(E / 8) * tid + h];
    sw[4 * h] = s4.x;
    sw[4 * h + 1] = s4.y;
    sw[4 * h + 2] = s4.z;
    sw[4 * h + 3] = s4.w;
  }
  // The sum up to the thread's first row end is its head, what follows its
  // last row end (everything, if no row ends here) its tail; a row between two
  // ends is complete.
  V acc = V(0), head = V(0);
  unsigned first = kNoRow;
#pragma unroll
  for (int j = 0; j < E; ++j) {
    acc = fma_v<V>(v[j], xv[j], acc);  // outside the branch: one FP64 instruction for the whole warp
    const unsigned r = (sw[j >> 1] >> (16 * (j & 1))) & 0xffffu;
    if (r != kNoRow) {
      if (first != kNoRow) {
        y[x0 + r] = acc;
      } else {
        head = acc;
        first = r;
      }
      acc = V(0);
    }
  }
  s_tail[tid] = acc;
  s_head[tid] = head;
  s_first[tid] = (unsigned short)first;
  const unsigned open = __ballot_sync(kFull, first == kNoRow && q < end);
  unsigned run = open;  // more than kReach threads in a row without a row end?
#pragma unroll
  for (int i = 1; i <= kReach; ++i) run &= open >> i;

  // 3. carries between threads.  Rows of a few threads each: every thread
  // walks back from its first row end.
  if (!__syncthreads_or(run != 0)) {
    const bool last = q < end && q + E >= end;
    if (first != kNoRow || last) {
      V s = first != kNoRow ? head : acc;
      for (int t = tid - 1; t >= 0; --t) {
        s += s_tail[t];
        if (s_first[t] != kNoRow) break;
      }
      if (first != kNoRow) y[x0 + first] = s;
      if (last) {
        carry_row[tile] = x0 + nrows;
        carry_val[tile] = first != kNoRow ? acc : s;
      }
    }
    if (tid == 0 && end == lead) {
      carry_row[tile] = x0 + nrows;
      carry_val[tile] = V(0);
    }
    return;
  }

  // Longer rows: by one warp of the tile (not the same one in each); a lane
  // takes the carries of K threads in a row.
  const int warps = (int)(blockDim.x >> 5), turn = tile & 3;
  if ((tid >> 5) != (turn < warps ? turn : 0)) return;
  if (warps == kRake) {
    // The default tile: everything a lane needs in a few vector loads.
    V tail[kRake], head4[kRake];
    unsigned short r4[kRake];
    rake_load(s_tail + lane * kRake, tail);
    rake_load(s_first + lane * kRake, r4);
    rake_load(s_head + lane * kRake, head4);
    bool ends = r4[0] != kNoRow;
    V sum = tail[0];
#pragma unroll
    for (int k = 1; k < kRake; ++k) {
      const bool f = r4[k] != kNoRow;
      ends |= f;
      sum = (f ? V(0) : sum) + tail[k];
    }
    sum = rake_scan(sum, ends, lane);
    if (lane == 31) {
      carry_row[tile] = x0 + nrows;
      carry_val[tile] = sum;
    }
    sum = __shfl_up_sync(kFull, sum, 1);
    if (lane == 0) sum = V(0);
#pragma unroll
    for (int k = 0; k < kRake; ++k) {
      const bool f = r4[k] != kNoRow;
      sum += f ? head4[k] : tail[k];
      if (f) {
        y[x0 + r4[k]] = sum;
        sum = tail[k];
      }
    }
    return;
  }
  const int K = warps, t0 = lane * K;
  bool ends = false;
  V sum = V(0);
  for (int k = 0; k < K; ++k) {
    const bool f = s_first[t0 + k] != kNoRow;
    ends |= f;
    sum = (f ? V(0) : sum) + s_tail[t0 + k];
  }
  sum = rake_scan(sum, ends, lane);
  if (lane == 31) {
    carry_row[tile] = x0 + nrows;
    carry_val[tile] = sum;
  }
  sum = __shfl_up_sync(kFull, sum, 1);
  if (lane == 0) sum = V(0);
  for (int k = 0; k < K; ++k) {
    const unsigned r = s_first[t0 + k];
    const V tail = s_tail[t0 + k];
    sum += r != kNoRow ? s_head[t0 + k] : tail;
    if (r != kNoRow) {
      y[x0 + r] = sum;
      sum = tail;
    }
  }
}

// 4. cross-tile carries: the first tile of each run of tiles that stopped in
// the same row adds the run's carries to that row.  A run of up to four tiles
// is summed by its thread; a longer one (a row of many tiles) by the thread's
// warp, lane l taking tiles l, l + 32, ... of the run, joined by a fixed xor
// tree, so a hub row costs a few loads in a row instead of one per tile.
template <typename V, typename Off>
__global__ void mp_fixup_kernel(const Off* carry_row, const V* carry_val, long long num_tiles, Off n_rows, V* y) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kShort = 4;
  release_next();
  wait_for_previous();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  Off r = n_rows;
  bool head = false, longer = false;
  if (t < num_tiles) {
    r = carry_row[t];
    head = r < n_rows && (t == 0 || carry_row[t - 1] != r);
    longer = head && t + kShort < num_tiles && carry_row[t + kShort] == r;
  }
  if (head && !longer) {
    V s = V(0);
#pragma unroll
    for (int u = 0; u < kShort; ++u)
      if (t + u < num_tiles && carry_row[t + u] == r) s += carry_val[t + u];
    y[r] += s;
  }
  for (unsigned m = __ballot_sync(kFull, longer); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    const long long t0 = t - lane + src;
    const Off row = __shfl_sync(kFull, r, src);
    V s = V(0);
    for (long long u = t0 + lane;; u += 32) {
      const bool in = u < num_tiles && carry_row[u] == row;
      if (in) s += carry_val[u];
      if (!__all_sync(kFull, in)) break;  // the run is contiguous: it ends here
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(kFull, s, off);
    if (lane == 0) y[row] += s;
  }
}

template <typename V, typename Off, int T, int B>
bool launch_tiles(const MpMatrix& m, int threads, const void* x, void* y, cudaStream_t s) {
  auto kern = mp_spmv_kernel<V, Off, T, B>;
  // A few KB of shared memory per CTA: leave the rest of the array to L1, which
  // serves the x gathers.
  static std::atomic<unsigned long long> configured{0};  // per instantiation, per device
  if (!once_per_device(configured, [&] {
        return VNEC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 32));
      }))
    return false;
  if (m.num_tiles > 0x7fffffffLL) {
    set_error("merge-path: tile count exceeds the grid limit");
    return false;
  }
  const bool vec = ((reinterpret_cast<uintptr_t>(m.col) | reinterpret_cast<uintptr_t>(m.val)) & 31) == 0;
  const size_t smem = (size_t)threads * ((E + 1) * sizeof(unsigned short) + 2 * sizeof(V));
  if (m.in_place)
    return launch_chained(kern, (unsigned)m.num_tiles, threads, smem, s, static_cast<const Off*>(m.row_end), m.col,
                          static_cast<const V*>(m.val), static_cast<const V*>(x), static_cast<V*>(y),
                          static_cast<const Off*>(m.tile_row), static_cast<const Off*>(m.tile_nz), (Off)m.nnz, vec,
                          static_cast<Off*>(m.carry_row), static_cast<V*>(m.carry_val));
  kern<<<(unsigned)m.num_tiles, threads, smem, s>>>(
      static_cast<const Off*>(m.row_end), m.col, static_cast<const V*>(m.val), static_cast<const V*>(x),
      static_cast<V*>(y), static_cast<const Off*>(m.tile_row), static_cast<const Off*>(m.tile_nz), (Off)m.nnz, vec,
      static_cast<Off*>(m.carry_row), static_cast<V*>(m.carry_val));
  return VNEC_CUDA(cudaGetLastError());
}

template <typename V, typename Off>
bool launch_mp(const MpMatrix& m, const void* x, void* y, cudaStream_t s, cudaEvent_t* ev) {
  if (ev && !VNEC_CUDA(cudaEventRecord(ev[0], s))) return false;
  const int threads = tile_threads((int)m.shape.items_per_tile());
  if (threads > kMaxTileThreads) {
    set_error("merge-path: unsupported tile shape");
    return false;
  }
  // 40 warps of an SM for FP64 (48 registers a thread), 64 for FP32: FP64 at 48
  // (40 registers, which spill) is 6% faster to 13% slower, at 36 up to 12%
  // slower; FP32 slows down by 7% at 48 warps and by 15% at 40.
  constexpr int kB = sizeof(V) == 8 ? 10 : 16;
  if (!(threads <= 128   ? launch_tiles<V, Off, 128, kB>(m, threads, x, y, s)
        : threads <= 256 ? launch_tiles<V, Off, 256, kB / 2>(m, threads, x, y, s)
                         : launch_tiles<V, Off, kMaxTileThreads, sizeof(V) == 8 ? 3 : 4>(m, threads, x, y, s)))
    return false;
  if (ev && !VNEC_CUDA(cudaEventRecord(ev[1], s))) return false;
  const int fb = 256;
  long long fg = (m.num_tiles + fb - 1) / fb;
  if (!launch_chained(mp_fixup_kernel<V, Off>, (unsigned)fg, fb, 0, s, static_cast<const Off*>(m.carry_row),
                      static_cast<const V*>(m.carry_val), (long long)m.num_tiles, (Off)m.n_rows, static_cast<V*>(y)))
    return false;
  if (ev && !VNEC_CUDA(cudaEventRecord(ev[2], s))) return false;
  return true;
}

}  // namespace

bool mp_partition(const MpMatrix& m, cudaStream_t s) {
  long long ipc = m.shape.items_per_tile();
  const int b = 256;
  long long g = (m.num_tiles + 1 + b - 1) / b;
  if (m.wide) {
    mp_partition_kernel<long long><<<(unsigned)g, b, 0, s>>>(
        static_cast<const long long*>(m.row_end), (long long)m.n_rows, (long long)m.nnz, ipc, m.num_tiles,
        static_cast<long long*>(const_cast<void*>(m.tile_row)), static_cast<long long*>(const_cast<void*>(m.tile_nz)));
  } else {
    mp_partition_kernel<int><<<(unsigned)g, b, 0, s>>>(
        static_cast<const int*>(m.row_end), (int)m.n_rows, (int)m.nnz, ipc, m.num_tiles,
        static_cast<int*>(const_cast<void*>(m.tile_row)), static_cast<int*>(const_cast<void*>(m.tile_nz)));
  }
  return VNEC_CUDA(cudaGetLastError());
}

bool mp_spmv(const MpMatrix& m, MpForm form, const void* x, void* y, cudaStream_t s, cudaEvent_t* ev) {
  if (m.n_rows == 0) return true;
  switch (form) {
    case MpForm::kF64:
      return m.wide ? launch_mp<double, long long>(m, x, y, s, ev) : launch_mp<double, int>(m, x, y, s, ev);
    case MpForm::kF32:
      return m.wide ? launch_mp<float, long long>(m, x, y, s, ev) : launch_mp<float, int>(m, x, y, s, ev);
  }
  set_error("merge-path: unknown value form");
  return false;
}

}  // namespace vnec

// ---------------------------------------------------------------------------
// Allocation-free entry point: SpB_mxv_csr_noalloc_ext.
//
// Some callers cannot let a library allocate device memory on their behalf:
// hosts whose device memory is handed out entirely by their own pool
// allocator (the library could not obtain more), and latency-critical loops
// in which a cudaMalloc/cudaFree and the device synchronisation it implies
// are not acceptable.  For them this entry point runs the FP64 merge-path
// kernel (256 threads, 2,040 merge items per tile) on CSR arrays the caller
// already holds in device memory, and keeps its scratch — the merge
// coordinates of each tile and each tile's carry-out — in the fixed array
// below, which every device that loads this library holds until the process
// exits.
// ---------------------------------------------------------------------------
namespace vnec {
namespace {

constexpr MpShape kNaShape{256, kMpPlaces};
// Scratch capacity: 2^18 tiles, 5,242,888 bytes.  The accepted size, n_rows + nnz
// <= 469,762,048, takes 230,276 of them.
constexpr long long kNaMaxTiles = 1LL << 18;
constexpr long long kNaMaxItems = 469762048;
static_assert((kNaMaxItems + kNaShape.items_per_tile() - 1) / kNaShape.items_per_tile() <= kNaMaxTiles,
              "the scratch holds every accepted size");
constexpr size_t kNaTileRowOff = 0;
constexpr size_t kNaTileNzOff = kNaTileRowOff + 4 * (kNaMaxTiles + 1);
constexpr size_t kNaCarryRowOff = kNaTileNzOff + 4 * (kNaMaxTiles + 1);
constexpr size_t kNaCarryValOff = kNaCarryRowOff + 4 * kNaMaxTiles;
constexpr size_t kNaBytes = kNaCarryValOff + 8 * kNaMaxTiles;
static_assert(kNaCarryValOff % 8 == 0, "carry values must be 8-byte aligned");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

// Identity of the calling thread's current CUDA context: its driver-assigned
// id, unique for the life of the process (cuCtxGetId), reached through the
// runtime's driver entry points so the library needs no link against the
// driver library.  False when the driver lacks these calls or no context is
// current yet.
using CtxGetCurrentFn = int (*)(void**);
using CtxGetIdFn = int (*)(void*, unsigned long long*);
bool current_context_id(unsigned long long* id) {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<CtxGetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(f);
  });
  if (!get_current || !get_id) return false;
  void* ctx = nullptr;
  if (get_current(&ctx) != 0 || !ctx) return false;
  return get_id(ctx, id) == 0;
}

// Device address of g_noalloc_scratch in the current context.  In host code
// the symbol is only a host-side stand-in, so the address is looked up with
// cudaGetSymbolAddress the first time a context calls and cached under that
// context's id: a device reset or a caller's own driver context gets a new id
// and therefore its own lookup, never a stale address.  Where the context id
// cannot be read, the address is looked up on every call.
bool noalloc_scratch(unsigned char** out) {
  struct Entry {
    unsigned long long ctx;
    unsigned char* addr;
  };
  static std::mutex mu;
  static Entry cache[64] = {};
  static int next = 0;
  unsigned long long id = 0;
  bool have_id = current_context_id(&id);
  if (have_id) {
    std::lock_guard<std::mutex> g(mu);
    for (const Entry& e : cache)
      if (e.addr && e.ctx == id) {
        *out = e.addr;
        return true;
      }
  }
  void* p = nullptr;
  if (!VNEC_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch))) return false;
  if (!p) {
    set_error("SpB_mxv_csr_noalloc_ext: no device address for the fixed scratch array");
    return false;
  }
  if (!have_id) have_id = current_context_id(&id);  // the lookup made the primary context current
  if (have_id) {
    std::lock_guard<std::mutex> g(mu);
    cache[next] = Entry{id, static_cast<unsigned char*>(p)};
    next = (next + 1) % 64;
  }
  *out = static_cast<unsigned char*>(p);
  return true;
}

}  // namespace
}  // namespace vnec

extern "C" SpB_Info SpB_mxv_csr_noalloc_ext(int64_t n_rows, int64_t n_cols, int64_t nnz, const int32_t* d_row_ptr,
                                            const int32_t* d_col, const double* d_val, const double* d_x,
                                            double* d_y, void* stream) {
  using namespace vnec;
  clear_error();
  if (n_rows < 0 || n_cols < 0 || nnz < 0) {
    set_error("SpB_mxv_csr_noalloc_ext: negative size");
    return SpB_FAILURE;
  }
  const long long ipc = kNaShape.items_per_tile();
  // Each size is checked on its own before the sum is formed, so huge
  // arguments cannot overflow it.
  if (n_rows > kNaMaxItems || nnz > kNaMaxItems || n_rows + nnz > kNaMaxItems) {
    set_error("SpB_mxv_csr_noalloc_ext: n_rows + nnz exceeds the allocation-free limit of 469,762,048 "
              "(its fixed scratch holds 262,144 tiles); use a plan (SpB_VNEC_plan_ext) instead");
    return SpB_FAILURE;
  }
  if (n_cols > INT32_MAX) {
    set_error("SpB_mxv_csr_noalloc_ext: n_cols exceeds the int32 column range");
    return SpB_FAILURE;
  }
  const long long tiles = (n_rows + nnz + ipc - 1) / ipc;
  if (n_rows == 0) return SpB_SUCCESS;
  if (!d_row_ptr || !d_y || (nnz > 0 && (!d_col || !d_val || !d_x))) {
    set_error("SpB_mxv_csr_noalloc_ext: NULL device array");
    return SpB_FAILURE;
  }
  unsigned char* scratch = nullptr;
  if (!noalloc_scratch(&scratch)) return SpB_FAILURE;
  MpMatrix m;
  m.n_rows = n_rows;
  m.n_cols = n_cols;
  m.nnz = nnz;
  m.wide = false;
  m.row_end = d_row_ptr + 1;
  m.col = d_col;
  m.val = d_val;
  m.tile_row = scratch + kNaTileRowOff;
  m.tile_nz = scratch + kNaTileNzOff;
  m.carry_row = scratch + kNaCarryRowOff;
  m.carry_val = scratch + kNaCarryValOff;
  m.num_tiles = tiles;
  m.shape = kNaShape;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // Every scratch word a launch reads is written earlier in the same call
  // (coordinates by the partition kernel, carries by the tile kernel), so
  // nothing needs clearing between calls.
  if (!mp_partition(m, s)) return SpB_FAILURE;
  return mp_spmv(m, MpForm::kF64, d_x, d_y, s) ? SpB_SUCCESS : SpB_FAILURE;
}
