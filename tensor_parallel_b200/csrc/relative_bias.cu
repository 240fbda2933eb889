// Relative-position score bias: out[h, i, j] = table[bucket(j - i), h], and the gradient of the table.
// The bias of a (query, key) pair depends on their distance only, so the bucket of each of the queries + keys - 1 distances is
// computed once by the caller (`buckets`, indexed by d = j - i + queries - 1) and nothing of [queries, keys] size is ever
// looked up, permuted or sorted:
//   forward  : bound by the one write of the bias; a CTA stages the values of the distances its tile spans in shared memory.
//   backward : bound by the one read of the gradient; threads own diagonals (consecutive threads, consecutive addresses), add
//              them up over a chunk of rows, and the CTA folds its diagonals into their buckets.  One fp32 partial table per
//              chunk, no atomics.
// The buckets themselves: one kernel, where the same over tensors is 14 (27 us for 1023 distances, and their launches).
// 32 heads x 512 x 512: 7 us and 12 us, where the lookup of every pair, its permutation, and the sort behind the embedding
// gradient took about 450 us.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "ptx_sm100.cuh"
#include "tpb_api.h"

namespace tpb {

typedef __nv_bfloat16 bf16;
constexpr int RB_THREADS = 128;
constexpr int RB_COLS = RB_THREADS * 8;  // columns of a forward tile
constexpr int RB_ROWS = 16;
constexpr int RB_BWD_THREADS = 256;
constexpr int RB_BWD_ROWS = 64;          // rows per partial table
constexpr int RB_DIAGS = 1024;           // diagonals folded at a time

__device__ __forceinline__ float rb_float(bf16 x) { return __bfloat162float(x); }
__device__ __forceinline__ float rb_float(float x) { return x; }
__device__ __forceinline__ void rb_nan(bf16& x) { x = __ushort_as_bfloat16(0x7FFF); }
__device__ __forceinline__ void rb_nan(float& x) { x = __int_as_float(0x7FFFFFFF); }

// A bucket that is no row of the table is not looked up: its distance gets NaN, and the status word says so.
template <typename T>
__global__ void __launch_bounds__(RB_THREADS)
relative_bias_kernel(const T* __restrict__ table, const int64_t* __restrict__ buckets, T* __restrict__ out, int heads, int queries, int keys,
                     int n_buckets, uint32_t* status) {
  __shared__ T vals[RB_COLS + RB_ROWS];
  const int h = blockIdx.z, i0 = blockIdx.y * RB_ROWS, j0 = blockIdx.x * RB_COLS;
  const int rows = min(RB_ROWS, queries - i0), cols = min(RB_COLS, keys - j0);
  const int d0 = j0 - (i0 + rows - 1) + queries - 1;  // smallest distance index of the tile
  for (int e = threadIdx.x; e < cols + rows - 1; e += RB_THREADS) {
    const int64_t b = buckets[d0 + e];
    if (uint64_t(b) < uint64_t(n_buckets)) {
      vals[e] = table[b * heads + h];
    } else {
      rb_nan(vals[e]);
      atomicMax(status, uint32_t(STATUS_BAD_ARG));
    }
  }
  __syncthreads();
  const int c = threadIdx.x * 8;
  if (c >= cols) return;
  const bool vec = sizeof(T) == 2 ? (keys & 7) == 0 : (keys & 3) == 0;  // (16-byte aligned rows; the base is)
  for (int r = 0; r < rows; ++r) {
    T* dst = out + ((long long)h * queries + i0 + r) * keys + j0 + c;
    const T* src = vals + c + rows - 1 - r;
    if (vec && c + 8 <= cols) {
      __align__(16) T v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = src[u];
#pragma unroll
      for (int u = 0; u < int(sizeof(T) / 2); ++u) reinterpret_cast<uint4*>(dst)[u] = reinterpret_cast<const uint4*>(v)[u];
    } else {
      for (int u = 0; u < 8 && c + u < cols; ++u) dst[u] = src[u];
    }
  }
}

// partial: fp32 [ceil(queries / RB_BWD_ROWS)][n_buckets][heads]
template <typename T>
__global__ void __launch_bounds__(RB_BWD_THREADS)
relative_bias_bwd_kernel(const T* __restrict__ grad, const int64_t* __restrict__ buckets, float* __restrict__ partial, int heads, int queries,
                         int keys, int n_buckets) {
  __shared__ float diag[RB_DIAGS];
  __shared__ int which[RB_DIAGS];
  __shared__ float fold[RB_BWD_THREADS];
  const int h = blockIdx.y, i0 = blockIdx.x * RB_BWD_ROWS;
  const int rows = min(RB_BWD_ROWS, queries - i0), diags = keys + rows - 1;
  const int d0 = queries - 1 - (i0 + rows - 1);  // distance index of diagonal 0 of this chunk: j = e - (rows - 1) + r
  const T* g = grad + ((long long)h * queries + i0) * keys;
  float* table = partial + (long long)blockIdx.x * n_buckets * heads + h;
  for (int e0 = 0; e0 < diags; e0 += RB_DIAGS) {
    const int n = min(RB_DIAGS, diags - e0);
    for (int e = threadIdx.x; e < n; e += RB_BWD_THREADS) {
      const int j0 = e0 + e - (rows - 1);  // column of row 0 of the chunk on this diagonal
      const int r_lo = max(0, -j0), r_hi = min(rows, keys - j0);
      float s = 0.f;
#pragma unroll 8
      for (int r = r_lo; r < r_hi; ++r) s += rb_float(g[(long long)r * keys + j0 + r]);
      diag[e] = s;
      const int64_t b = buckets[d0 + e0 + e];
      which[e] = uint64_t(b) < uint64_t(n_buckets) ? int(b) : -1;  // (reported by the forward)
    }
    __syncthreads();
    for (int b0 = 0; b0 < n_buckets; b0 += 32) {  // 32 buckets x 8 slices of the diagonals
      const int b = b0 + (threadIdx.x & 31), slice = threadIdx.x >> 5;
      float s = 0.f;
      for (int e = slice; e < n; e += RB_BWD_THREADS / 32) s += which[e] == b ? diag[e] : 0.f;
      fold[threadIdx.x] = s;
      __syncthreads();
      if (threadIdx.x < 32 && b < n_buckets) {
        float t = 0.f;
        for (int k = 0; k < RB_BWD_THREADS / 32; ++k) t += fold[k * 32 + threadIdx.x];
        float* dst = table + (long long)b * heads;
        *dst = e0 ? *dst + t : t;
      }
      __syncthreads();
    }
  }
}

// Bucket of each of `count` consecutive distances from `first` up, as relative position embeddings count them: half of the buckets per direction
// (bidirectional) or all for distances up to 0; exact up to max_exact, logarithmic above.  The fp32 expression is the one that the same
// steps over tensors evaluate, a division by a number being a multiplication by its reciprocal (rounded to fp32 once), so that the buckets are equal.
__global__ void relative_buckets_kernel(int64_t* __restrict__ out, long long first, long long count, int bidirectional, int per_direction, int max_exact,
                                        float inv_exact, float inv_log, float log_buckets) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= count) return;
  const long long d = first + i;
  const long long far = bidirectional ? (d < 0 ? -d : d) : (d < 0 ? -d : 0);
  long long bucket = far;
  if (far >= max_exact) {
    const float steps = __fmul_rn(__fmul_rn(logf(__fmul_rn(fmaxf(float(far), 1.f), inv_exact)), inv_log), log_buckets);
    const long long large = max_exact + (long long)steps;
    bucket = large < per_direction - 1 ? large : per_direction - 1;
  }
  out[i] = bucket + (bidirectional && d > 0 ? per_direction : 0);
}

}  // namespace tpb

using namespace tpb;

// table: [n_buckets, heads] contiguous; buckets: int64 [queries + keys - 1]; out: [heads, queries, keys]; dtype: 0 = bf16, 1 = fp32.
// status: device word that becomes STATUS_BAD_ARG if a bucket is not in [0, n_buckets).
extern "C" int tpb_relative_bias(const void* table, const int64_t* buckets, void* out, int heads, int queries, int keys, int n_buckets, int dtype,
                                 void* status, void* stream_) {
  if (!table || !buckets || !out || !status || heads <= 0 || queries <= 0 || keys <= 0 || n_buckets <= 0 || heads > 65535 ||
      (queries + RB_ROWS - 1) / RB_ROWS > 65535)
    return TPB_ERR_ARG;
  if (reinterpret_cast<uintptr_t>(out) & 15) return TPB_ERR_ALIGN;
  const dim3 grid((keys + RB_COLS - 1) / RB_COLS, (queries + RB_ROWS - 1) / RB_ROWS, heads);
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  uint32_t* st = static_cast<uint32_t*>(status);
  if (dtype == 0)
    relative_bias_kernel<bf16><<<grid, RB_THREADS, 0, s>>>((const bf16*)table, buckets, (bf16*)out, heads, queries, keys, n_buckets, st);
  else
    relative_bias_kernel<float><<<grid, RB_THREADS, 0, s>>>((const float*)table, buckets, (float*)out, heads, queries, keys, n_buckets, st);
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

// Rows of partial tables that tpb_relative_bias_bwd writes.
extern "C" int tpb_relative_bias_parts(int queries) { return (queries + RB_BWD_ROWS - 1) / RB_BWD_ROWS; }

// grad: [heads, queries, keys] contiguous; buckets as above, those out of range contribute nothing; partial: fp32 [tpb_relative_bias_parts(queries)][n_buckets][heads], to be summed by the caller.
extern "C" int tpb_relative_bias_bwd(const void* grad, const int64_t* buckets, float* partial, int heads, int queries, int keys, int n_buckets, int dtype,
                                     void* stream_) {
  if (!grad || !buckets || !partial || heads <= 0 || queries <= 0 || keys <= 0 || n_buckets <= 0 || heads > 65535) return TPB_ERR_ARG;
  const dim3 grid(tpb_relative_bias_parts(queries), heads);
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  if (dtype == 0)
    relative_bias_bwd_kernel<bf16><<<grid, RB_BWD_THREADS, 0, s>>>((const bf16*)grad, buckets, partial, heads, queries, keys, n_buckets);
  else
    relative_bias_bwd_kernel<float><<<grid, RB_BWD_THREADS, 0, s>>>((const float*)grad, buckets, partial, heads, queries, keys, n_buckets);
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

// out: int64 [count], the buckets of distances first, first + 1, ...; buckets: of both directions together.  Needs buckets for at least one exact
// distance per direction and a max_distance beyond the exact ones.
extern "C" int tpb_relative_buckets(int64_t* out, long long first, long long count, int bidirectional, int buckets, int max_distance, void* stream_) {
  const int per_direction = bidirectional ? buckets / 2 : buckets, max_exact = per_direction / 2;
  if (!out || count <= 0 || count > (1ll << 31) || max_exact < 1 || max_distance <= max_exact) return TPB_ERR_ARG;
  const float inv_log = float(1.0 / log(double(max_distance) / double(max_exact))), inv_exact = float(1.0 / double(max_exact));
  relative_buckets_kernel<<<int((count + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream_)>>>(out, first, count, bidirectional, per_direction, max_exact,
                                                                                                 inv_exact, inv_log, float(per_direction - max_exact));
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}
