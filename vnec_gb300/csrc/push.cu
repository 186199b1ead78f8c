// Push-side sparse-matrix x sparse-vector product (SpMSpV, the operation the
// reference declares as SpB_vxm, OpenSparseBLAS.h:1940, without a body):
// y = A x for a sparse x given as (index, value) pairs, touching only the
// columns of A that x selects.  A is held as its CSC (the CSR of A^T); each
// entry of a selected column adds value * x_j into y with FP64 (FP32) atomics,
// so the order of the additions into one y entry varies from run to run
// (results agree to rounding, not bit for bit).  An index outside [0, n_cols)
// is skipped and recorded in a device status word.
//
// Split of the work.  A frontier of a power-law graph mixes columns of one
// entry with hubs of tens of thousands, so neither columns nor warps per
// column balance (plans of short columns only: push_columns_kernel).  The
// entries of x are dealt out to chunks of kChunk (entry i * chunks + c to chunk
// c, so that neighbouring hubs fall to different chunks); `parts` blocks share a
// chunk: each scans the chunk's column lengths into shared memory and takes an
// equal share of their sum, cut into one contiguous run per warp.  The scan is repeated by the chunk's blocks instead
// of handed from one launch to the next: it is three loads a thread, and calls
// on several streams share no scratch.
// What bounds it now: the L2's atomics, the ones on the lines of the hub rows
// above all (the first 16 rows, one line, of R-MAT 2^20 take 61,000 of a
// 50,000-vertex frontier's 7.9 M additions; adding hub rows up in shared memory
// first took 98 -> 80 us there, but 29 -> 33 with 5,000 vertices and 709 ->
// 1000 with a dense x).
// Measured (us, one warp per column before): R-MAT 2^20, frontiers of 64, 500,
// 5,000, 50,000 and 131,072 vertices reached along edges: 110 -> 10, 135 -> 13,
// 406 -> 29, 624 -> 98, 720 -> 176; dense x 1054 -> 709.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.h"
#include "push.h"

namespace vnec {
namespace {

constexpr int kChunk = 256;  // entries of x per chunk, threads per block
constexpr int kWarps = kChunk / 32;
constexpr int kUnroll = 4;   // column entries in flight per lane

// Blocks wanted in all: enough that a chunk with a hub column of tens of
// thousands of entries is shared by many (half or twice as many: within 5%).
constexpr long long kBlocks = 152LL * 16;
// ... but beyond one block an SM no more than give each at least this many
// entries, were the frontier's columns average and one the longest: every part
// scans its chunk anew (R-MAT 2^13, dense x: 19.6 -> 13.5 us; fewer parts for
// chunks that do not fill the GPU: 137 vertices of 2^16 9.2 -> 10.2).
constexpr long long kPartEntries = 256;

template <typename V>
__global__ void __launch_bounds__(kChunk)
push_kernel(long long nx, const int32_t* __restrict__ idx, const V* __restrict__ xval, const int64_t* __restrict__ cp,
            const int32_t* __restrict__ row, const V* __restrict__ val, long long n_cols, unsigned chunks,
            unsigned parts, V* __restrict__ y, int* __restrict__ status) {
  __shared__ long long s_off[kChunk + 1];  // entries of the chunk's columns before column i
  __shared__ long long s_src[kChunk];      // first entry of column i, less s_off[i]
  __shared__ V s_x[kChunk];
  __shared__ long long s_warp[kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned chunk = blockIdx.x / parts, part = blockIdx.x % parts;

  // The chunk's columns: lengths (0 for an index out of range or a zero of x),
  // scanned over the block.
  long long len = 0, begin = 0;
  V xj = V(0);
  const long long w = (long long)tid * chunks + chunk;
  if (w < nx) {
    const long long j = idx ? (long long)__ldg(idx + w) : w;
    if (j < 0 || j >= n_cols) {
      if (part == 0) atomicExch(status, 1);
    } else {
      xj = __ldg(xval + w);
      begin = __ldg(cp + j);
      const long long end = __ldg(cp + j + 1);
      if (xj != V(0)) len = end - begin;
    }
  }
  long long sum = len;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const long long up = __shfl_up_sync(0xffffffffu, sum, d);
    if (lane >= d) sum += up;
  }
  if (lane == 31) s_warp[warp] = sum;
  __syncthreads();
  long long before = 0;
#pragma unroll
  for (int i = 0; i < kWarps; ++i)
    if (i < warp) before += s_warp[i];
  const long long off = before + sum - len;
  s_off[tid] = off;
  s_src[tid] = begin - off;
  s_x[tid] = xj;
  if (tid == kChunk - 1) s_off[kChunk] = before + sum;
  __syncthreads();

  // This warp's run of the chunk's entries.
  const long long total = s_off[kChunk];
  const unsigned slot = part * kWarps + warp, slots = parts * kWarps;
  const long long p0 = total / slots * slot + min((long long)slot, total % slots);
  const long long p1 = p0 + total / slots + (slot < total % slots ? 1 : 0);
  long long p = p0 + lane;
  int c = 0;  // the last column that starts at or before p
  if (p < p1)
    for (int d = kChunk / 2; d > 0; d >>= 1)
      if (s_off[c + d] <= p) c += d;
  for (; p < p1; p += 32 * kUnroll) {
    long long src[kUnroll];
    V x[kUnroll], v[kUnroll];
    int r[kUnroll];
#pragma unroll
    for (int u = 0; u < kUnroll; ++u) {
      const long long q = p + 32 * u;
      src[u] = -1;
      if (q < p1) {
        while (s_off[c + 1] <= q) ++c;
        src[u] = s_src[c] + q;
        x[u] = s_x[c];
      }
    }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (src[u] >= 0) {
        r[u] = __ldcs(row + src[u]);
        v[u] = __ldcs(val + src[u]);
      }
#pragma unroll
    for (int u = 0; u < kUnroll; ++u)
      if (src[u] >= 0) atomicAdd(y + r[u], v[u] * x[u]);
  }
}

// One warp per column, for plans whose columns are all short: without hubs there
// is nothing to balance, and a warp has its column's entries after two dependent
// loads, where the scan costs a block four and two barriers.
template <typename V>
__global__ void __launch_bounds__(kChunk)
push_columns_kernel(long long nx, const int32_t* __restrict__ idx, const V* __restrict__ xval,
                    const int64_t* __restrict__ cp, const int32_t* __restrict__ row, const V* __restrict__ val,
                    long long n_cols, V* __restrict__ y, int* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const long long nw = (long long)gridDim.x * kWarps;
  for (long long w = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5); w < nx; w += nw) {
    const long long j = idx ? (long long)__ldg(idx + w) : w;
    if (j < 0 || j >= n_cols) {
      if (lane == 0) atomicExch(status, 1);
      continue;
    }
    const V xj = __ldg(xval + w);
    if (xj == V(0)) continue;
    const long long b = __ldg(cp + j), e = __ldg(cp + j + 1);
    for (long long p = b + lane; p < e; p += 32) atomicAdd(y + __ldg(row + p), __ldcs(val + p) * xj);
  }
}

// Columns one by one where none is longer than kShortColumn and there are enough of
// them to fill the GPU (else a chunk's blocks share a column: 33 columns of 300
// entries 10.3 us by warps, 8.3 shared).  The more columns, the more the scan
// gets out of full warps, and the sooner so the shorter they are.  us, shared ->
// by warps, FP64: 20 entries a column (lognormal rows), 4,000 columns 14.2 -> 8.3,
// 50,000 22.7 -> 16.4; 9 entries, 6,000 14.5 -> 8.0, 75,000 18.6 -> 18.5, 300,000
// 32.8 -> 47; 33 entries, 200,000 34.9 -> 47; 100 entries, 25,000 28.7 -> 22.6,
// 100,000 74.6 -> 63.5; 1 entry, 1,000 10.3 -> 9.7, 40,000 11.5 -> 13.6.
constexpr int64_t kShortColumn = 512;
bool by_columns(const PushMatrix& m, long long nx) {
  if (m.longest > kShortColumn || nx < 256) return false;
  return m.nnz >= 64 * m.n_cols || nx <= 16384 || (nx <= 131072 && m.nnz >= 8 * m.n_cols);
}

template <typename V>
bool launch(const PushMatrix& m, long long nx, const int32_t* idx, const void* xval, void* y, cudaStream_t s) {
  if (m.n_rows > 0 && !VNEC_CUDA(cudaMemsetAsync(y, 0, sizeof(V) * (size_t)m.n_rows, s))) return false;
  if (nx <= 0) return true;
  if (by_columns(m, nx)) {
    const long long grid = std::min<long long>((nx + kWarps - 1) / kWarps, 152LL * 32);
    push_columns_kernel<V><<<(unsigned)grid, kChunk, 0, s>>>(nx, idx, static_cast<const V*>(xval), m.col_ptr, m.row,
                                                            static_cast<const V*>(m.val), m.n_cols,
                                                            static_cast<V*>(y), m.status);
    return VNEC_CUDA(cudaGetLastError());
  }
  const long long chunks = (nx + kChunk - 1) / kChunk;
  const long long most = kChunk * (m.nnz / std::max<long long>(m.n_cols, 1) + 1) + m.longest;
  const long long want = std::max<long long>(152 / chunks, (most + kPartEntries - 1) / kPartEntries);
  const long long parts = std::max<long long>(1, std::min<long long>({kBlocks / chunks, 64, want}));
  if (chunks * parts > 0x7fffffffLL) {
    set_error("SpMSpV: too many entries of x for one launch");
    return false;
  }
  push_kernel<V><<<(unsigned)(chunks * parts), kChunk, 0, s>>>(
      nx, idx, static_cast<const V*>(xval), m.col_ptr, m.row, static_cast<const V*>(m.val), m.n_cols,
      (unsigned)chunks, (unsigned)parts, static_cast<V*>(y), m.status);
  return VNEC_CUDA(cudaGetLastError());
}

}  // namespace

bool push_spmspv(const PushMatrix& m, bool fp64, long long nx, const int32_t* idx, const void* xval, void* y,
                 cudaStream_t s) {
  return fp64 ? launch<double>(m, nx, idx, xval, y, s) : launch<float>(m, nx, idx, xval, y, s);
}

}  // namespace vnec
