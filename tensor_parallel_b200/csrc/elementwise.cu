// Memory-bound operators: RMSNorm / LayerNorm (forward + backward, optional fused residual add),
// rotary embedding, gated / plain activations (forward + backward), embedding gather, fused AdamW,
// dtype casts.  All kernels move data with 16-byte vector accesses and keep a row resident in
// registers between the statistics pass and the normalisation pass, so every tensor is read once.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <atomic>
#include <type_traits>

#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "tpb_api.h"

namespace tpb {

typedef __nv_bfloat16 bf16;

template <typename T> struct Vec8 {};  // 8 elements of T <-> 8 floats
template <> struct Vec8<bf16> {
  static __device__ __forceinline__ void load(const bf16* p, float (&v)[8]) {
    uint4 u = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
  static __device__ __forceinline__ void store(bf16* p, const float (&v)[8]) {
    uint4 u;
    uint32_t* w = &u.x;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(p) = u;
  }
};
template <> struct Vec8<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[8]) {
    float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[8]) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  }
};

template <typename T> __device__ __forceinline__ float to_f(T x);
template <> __device__ __forceinline__ float to_f<bf16>(bf16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_f<float>(float x) { return x; }
template <typename T> __device__ __forceinline__ T from_f(float x);
template <> __device__ __forceinline__ bf16 from_f<bf16>(float x) { return __float2bfloat16(x); }
template <> __device__ __forceinline__ float from_f<float>(float x) { return x; }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-wide sums of two values, or (not BOTH) of the second only, whose shuffles no compiler takes out; blockDim.x <= 1024
template <bool BOTH>
__device__ __forceinline__ void block_sum2(float& a, float& b) {
  __shared__ float sa[32], sb[32];
  if (BOTH) a = warp_sum(a);
  b = warp_sum(b);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) {
    if (BOTH) sa[warp] = a;
    sb[warp] = b;
  }
  __syncthreads();
  if (BOTH) a = warp_sum(lane < nw ? sa[lane] : 0.f);
  b = warp_sum(lane < nw ? sb[lane] : 0.f);
}

template <typename T> struct Raw8 { uint4 u[sizeof(T) / 2]; };  // 8 elements as they lie in memory
template <typename T> __device__ __forceinline__ Raw8<T> load_raw(const T* p) {
  Raw8<T> r;
#pragma unroll
  for (int i = 0; i < int(sizeof(T) / 2); ++i) r.u[i] = reinterpret_cast<const uint4*>(p)[i];
  return r;
}
__device__ __forceinline__ void unpack(const Raw8<bf16>& r, float (&v)[8]) {
  const uint32_t w[4] = {r.u[0].x, r.u[0].y, r.u[0].z, r.u[0].w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ void pack(const float (&v)[8], Raw8<float>& r) {
  r.u[0] = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
  r.u[1] = make_uint4(__float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7]));
}
__device__ __forceinline__ void unpack(const Raw8<float>& r, float (&v)[8]) {
  const uint32_t w[8] = {r.u[0].x, r.u[0].y, r.u[0].z, r.u[0].w, r.u[1].x, r.u[1].y, r.u[1].z, r.u[1].w};
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(w[i]);
}

// ------------------------------------------------------------------------------------------------
// Norms.  One CTA per row; a thread holds up to MAXV vectors of 8 elements (cols <= blockDim*8*MAXV).
// mode 0 = RMSNorm (no mean, no bias), mode 1 = LayerNorm.
// If residual != null:  h = x + residual is normalised and also written to sum_out.
// ------------------------------------------------------------------------------------------------
constexpr int NORM_THREADS = 256;
constexpr int NORM_MAXV = 8;  // cols <= 16384

// CTAs of a row each that an SM is to hold, at least: the most that registers allow without spills.  A row is bound by the chain load - sums - store, so
// that rows in flight are what counts: RMSNorm bf16 8192 x 5120 with six / five CTAs 29.8 / 31.2 us, 8192 x 8192 with five / four 43.6 / 46.7; LayerNorm
// 4096 wide spills with six (600 rows 3.86 -> 4.33), 5120 wide loses with four (8192 rows 41.9 -> 44.6), 8192 wide with three (56 -> 63).
template <typename T, int MODE, int MAXV, bool RES>
constexpr int norm_row_ctas_per_sm() {
  if (RES || sizeof(T) == 4) return 1;
  if (MODE == 0) return MAXV <= 2 ? 8 : MAXV == 3 ? 6 : MAXV == 4 ? 5 : 4;
  return MAXV == 1 ? 8 : MAXV <= 3 ? 5 : 4;
}

// MAXV = vectors of 8 elements a thread may hold (cols <= 256 * 8 * MAXV).  RES = there is a residual; without one the row waits for its sums as it lies
// in memory: 32 registers a thread for up to 4096 bf16 columns, so that eight rows are in flight per SM, and the weights are fetched before the sums are
// known.  RMSNorm bf16 8192 x 4096 29.6 -> 22.7 us (5.9 TB/s), 1000 x 4096 in L2 / in memory 5.1 -> 3.5 / 6.8 -> 5.1, 20 x 4096 2.5 -> 2.1; 8192 x 12288 148 -> 63.
template <typename T, int MODE, int MAXV, bool RES>
__global__ void __launch_bounds__(NORM_THREADS, norm_row_ctas_per_sm<T, MODE, MAXV, RES>())
norm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ residual, const T* __restrict__ weight,
                const T* __restrict__ bias, T* __restrict__ out, T* __restrict__ sum_out, float* __restrict__ rstd_out,
                float* __restrict__ mean_out, int cols, float eps) {
  constexpr bool EARLY = !RES && MAXV <= 2;  // weights before the sums, where registers allow it
  pdl_wait();
  const size_t row = blockIdx.x;
  const T* xr = x + row * cols;
  const int nvec = cols >> 3;
  Raw8<typename std::conditional<RES, float, T>::type> held[MAXV];
  Raw8<T> wr[EARLY ? MAXV : 1];
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int vi = threadIdx.x + i * NORM_THREADS;
    if (vi < nvec) {
      if constexpr (RES) {
        float v[8], r[8];
        Vec8<T>::load(xr + vi * 8, v);
        Vec8<T>::load(residual + row * cols + vi * 8, r);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] += r[j];
        if (sum_out) {
          // round to the storage type first so that the statistics match what later kernels will read
          Vec8<T>::store(sum_out + row * cols + vi * 8, v);
          Vec8<T>::load(sum_out + row * cols + vi * 8, v);
        }
        pack(v, held[i]);
      } else {
        held[i] = load_raw(xr + vi * 8);
      }
    }
  }
  if constexpr (EARLY) {
#pragma unroll
    for (int i = 0; i < MAXV; ++i) {
      const int vi = threadIdx.x + i * NORM_THREADS;
      if (vi < nvec && weight) wr[i] = load_raw(weight + vi * 8);
    }
  }
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    if (int(threadIdx.x) + i * NORM_THREADS < nvec) {
      float v[8];
      unpack(held[i], v);
#pragma unroll
      for (int j = 0; j < 8; ++j) { s1 += v[j]; s2 += v[j] * v[j]; }
    }
  }
  block_sum2<MODE == 1>(s1, s2);
  const float inv_n = 1.f / float(cols);
  const float mean = MODE == 1 ? s1 * inv_n : 0.f;
  const float var = MODE == 1 ? fmaxf(s2 * inv_n - mean * mean, 0.f) : s2 * inv_n;
  const float rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0) {
    if (rstd_out) rstd_out[row] = rstd;
    if (mean_out) mean_out[row] = mean;
  }
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    const int vi = threadIdx.x + i * NORM_THREADS;
    if (vi < nvec) {
      float v[8], w[8], b[8], o[8];
      unpack(held[i], v);
      if constexpr (EARLY) { if (weight) unpack(wr[i], w); }
      else if (weight) Vec8<T>::load(weight + vi * 8, w);
      if (MODE == 1 && bias) Vec8<T>::load(bias + vi * 8, b);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float y = (v[j] - mean) * rstd;
        if (weight) y *= w[j];
        if (MODE == 1 && bias) y += b[j];
        o[j] = y;
      }
      Vec8<T>::store(out + row * cols + vi * 8, o);
    }
  }
}

// Backward: dx per row; the column sums for dweight / dbias go through one fp32 partial row per CTA, which
// norm_bwd_reduce_kernel adds up in a fixed order (deterministic, no atomics).  Memory-bound: x and dy are read and dx is
// written once.  A thread owns 8 columns (a CTA has as many threads as the row has vectors, so that its registers admit 1024
// threads per SM whatever the width) and walks rows blockIdx.x, + gridDim.x, ... with the column sums in registers.  Rows arrive through
// a ring of private slots in shared memory (cp.async; nobody reads another thread's slot), three rows ahead (fp32: two): one row ahead
// in registers kept 32 KB per SM in flight, too little for the latency of a loaded memory system.  RMSNorm 8192 x 4096 bf16 63 -> 48 us
// (4.2 TB/s), 8192 x 8192 122 -> 86; LayerNorm 1999 x 5120 fp32 44 -> 40 us, 8192 x 8192 fp32 201 -> 162; 20 x 4096 5.0 and 5.0.
constexpr int NORM_BWD_MAXC = 8192;  // 1024 threads

// The 8 columns of a thread in 16-byte chunks: bf16 one chunk, fp32 two, which lie blockDim.x chunks apart so that a warp's accesses are
// contiguous (cp.async goes past L1: chunks side by side would fetch every 32-byte sector twice).
template <typename T>
struct RowCols {
  static constexpr int CHUNKS = sizeof(T) / 2, WIDTH = 16 / sizeof(T);
  static __device__ __forceinline__ int at(int i) { return (threadIdx.x + i * blockDim.x) * WIDTH; }
  static __device__ __forceinline__ Raw8<T> load(const T* row, int cols) {
    Raw8<T> r;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) r.u[i] = at(i) < cols ? *reinterpret_cast<const uint4*>(row + at(i)) : make_uint4(0, 0, 0, 0);
    return r;
  }
  template <typename O>
  static __device__ __forceinline__ void store(O* row, int cols, const float (&v)[8]) {
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      if (at(i) >= cols) continue;
      if constexpr (CHUNKS == 1) Vec8<O>::store(row + at(0), v);
      else reinterpret_cast<float4*>(row)[threadIdx.x + i * blockDim.x] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
  }
};

// Private ring of a thread: STAGES slots of N row slices (8 elements each) in shared memory.  Slots are interleaved by 16-byte chunk, so
// that a warp's accesses are contiguous.
template <typename T, int N>
struct RowRing {
  static constexpr int STAGES = sizeof(T) == 2 && N == 2 ? 4 : 3;
  static constexpr int CHUNKS = RowCols<T>::CHUNKS;
  static size_t bytes(int threads) { return size_t(threads) * STAGES * N * CHUNKS * 16; }
  uint4* base;
  __device__ __forceinline__ uint4* slot(int stage, int n, int chunk) const {
    return base + ((stage * N + n) * CHUNKS + chunk) * blockDim.x + threadIdx.x;
  }
  __device__ __forceinline__ void fetch(int stage, int n, const T* row, int cols) const {
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i)
      if (RowCols<T>::at(i) < cols)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(slot(stage, n, i))), "l"(row + RowCols<T>::at(i)) : "memory");
  }
  __device__ __forceinline__ Raw8<T> get(int stage, int n, int cols) const {
    Raw8<T> r;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) r.u[i] = RowCols<T>::at(i) < cols ? *slot(stage, n, i) : make_uint4(0, 0, 0, 0);
    return r;
  }
  // one group per row, empty ones included: the row fetched STAGES - 1 groups ago has arrived
  static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  static __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 1) : "memory"); }
};

// Block-wide sums of two values per row, or (not BOTH) of the second only; one barrier per row: `turn` alternates between two sets of warp sums.
template <bool BOTH>
__device__ __forceinline__ void row_sum2(float2 (*warp_sums)[32], int turn, float& a, float& b) {
  if (BOTH) a = warp_sum(a);
  b = warp_sum(b);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  if (nw == 1) return;
  if (lane == 0) warp_sums[turn][warp] = make_float2(a, b);
  __syncthreads();
  const float2 w = lane < nw ? warp_sums[turn][lane] : make_float2(0.f, 0.f);
  if (BOTH) a = warp_sum(w.x);
  b = warp_sum(w.y);
}

template <typename T, int MODE>
__global__ void __launch_bounds__(1024)
norm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ weight,
                const float* __restrict__ rstd_in, const float* __restrict__ mean_in, T* __restrict__ dx,
                float* __restrict__ part_w, float* __restrict__ part_b, unsigned rows, int cols) {
  using Ring = RowRing<T, 2>;
  extern __shared__ uint4 norm_ring[];
  __shared__ float2 warp_sums[2][32];
  const Ring ring{norm_ring};
  float dw_acc[8], db_acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) { dw_acc[j] = 0.f; db_acc[j] = 0.f; }
  auto fetch = [&](int stage, unsigned row) {  // (rows unsigned: the row after the last may be beyond 2^31)
    if (row < rows) {
      ring.fetch(stage, 0, dy + size_t(row) * cols, cols);
      ring.fetch(stage, 1, x + size_t(row) * cols, cols);
    }
    Ring::commit();
  };
#pragma unroll
  for (int i = 0; i < Ring::STAGES - 1; ++i) fetch(i, blockIdx.x + i * gridDim.x);
  Raw8<T> wr;
  if (weight) wr = RowCols<T>::load(weight, cols);
  const float inv_n = 1.f / float(cols);
  unsigned row = blockIdx.x;
  float rstd = 0.f, mean = 0.f;
  if (row < rows) {
    rstd = rstd_in[row];
    if (MODE == 1) mean = mean_in[row];
  }
  for (int it = 0; row < rows; ++it) {
    const unsigned next = row + gridDim.x;
    fetch((it + Ring::STAGES - 1) % Ring::STAGES, row + (Ring::STAGES - 1) * gridDim.x);
    float rstd_next = 0.f, mean_next = 0.f;
    if (next < rows) {
      rstd_next = rstd_in[next];
      if (MODE == 1) mean_next = mean_in[next];
    }
    Ring::wait();
    float s1 = 0.f, s2 = 0.f;  // sum(g), sum(g * xhat)
    const Raw8<T> dr = ring.get(it % Ring::STAGES, 0, cols), xr = ring.get(it % Ring::STAGES, 1, cols);
    {
      float d[8], xv[8], w[8];
      unpack(dr, d);
      unpack(xr, xv);
      if (weight) unpack(wr, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (xv[j] - mean) * rstd;
        dw_acc[j] += d[j] * xh;
        db_acc[j] += d[j];
        const float g = weight ? d[j] * w[j] : d[j];
        s1 += g;
        s2 += g * xh;
      }
    }
    row_sum2<MODE == 1>(warp_sums, it & 1, s1, s2);
    const float c1 = MODE == 1 ? s1 * inv_n : 0.f;
    const float c2 = s2 * inv_n;
    {
      float d[8], xv[8], w[8], o[8];
      unpack(dr, d);
      unpack(xr, xv);
      if (weight) unpack(wr, w);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (xv[j] - mean) * rstd;
        const float g = weight ? d[j] * w[j] : d[j];
        o[j] = (g - c1 - xh * c2) * rstd;
      }
      RowCols<T>::store(dx + size_t(row) * cols, cols, o);
    }
    row = next;
    rstd = rstd_next;
    mean = mean_next;
  }
  if (part_w) RowCols<T>::store(part_w + size_t(blockIdx.x) * cols, cols, dw_acc);
  if (MODE == 1 && part_b) RowCols<T>::store(part_b + size_t(blockIdx.x) * cols, cols, db_acc);
}

// Forward without a residual: rows stream through the same rings; weight and bias stay in registers.  For narrow rows, which left threads of a
// CTA per row idle, fp32 rows, and few rows (norm_takes_row_cta).  LayerNorm 1999 x 5120 fp32 23.1 -> 17.7 us, 8192 x 1024 bf16 17.5 -> 10.7; RMSNorm
// 8192 x 256 bf16 11.3 -> 4.8.  bf16: CTAs for 2048 threads per SM; fp32: 1024 (2048: RMSNorm 8192 x 4096 46 -> 49, 8192 x 8192 81 -> 95 us).
template <typename T, int MODE>
__global__ void __launch_bounds__(1024, sizeof(T) == 2 && MODE == 0 ? 2 : 1)
norm_fwd_rows_kernel(const T* __restrict__ x, const T* __restrict__ weight, const T* __restrict__ bias, T* __restrict__ out,
                     float* __restrict__ rstd_out, float* __restrict__ mean_out, unsigned rows, int cols, float eps) {
  using Ring = RowRing<T, 1>;
  extern __shared__ uint4 norm_ring[];
  __shared__ float2 warp_sums[2][32];
  const Ring ring{norm_ring};
  auto fetch = [&](int stage, unsigned row) {
    if (row < rows) ring.fetch(stage, 0, x + size_t(row) * cols, cols);
    Ring::commit();
  };
  pdl_wait();
#pragma unroll
  for (int i = 0; i < Ring::STAGES - 1; ++i) fetch(i, blockIdx.x + i * gridDim.x);
  Raw8<T> wr, br;
  if (weight) wr = RowCols<T>::load(weight, cols);
  if (MODE == 1 && bias) br = RowCols<T>::load(bias, cols);
  const float inv_n = 1.f / float(cols);
  int it = 0;
  for (unsigned row = blockIdx.x; row < rows; ++it, row += gridDim.x) {
    fetch((it + Ring::STAGES - 1) % Ring::STAGES, row + (Ring::STAGES - 1) * gridDim.x);
    Ring::wait();
    float v[8], s1 = 0.f, s2 = 0.f;
    unpack(ring.get(it % Ring::STAGES, 0, cols), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s1 += v[j];
      s2 += v[j] * v[j];
    }
    row_sum2<MODE == 1>(warp_sums, it & 1, s1, s2);
    const float mean = MODE == 1 ? s1 * inv_n : 0.f;
    const float var = MODE == 1 ? fmaxf(s2 * inv_n - mean * mean, 0.f) : s2 * inv_n;
    const float rstd = rsqrtf(var + eps);
    if (threadIdx.x == 0) {
      if (rstd_out) rstd_out[row] = rstd;
      if (mean_out) mean_out[row] = mean;
    }
    float w[8], b[8], o[8];
    if (weight) unpack(wr, w);
    if (MODE == 1 && bias) unpack(br, b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float y = (v[j] - mean) * rstd;
      if (weight) y *= w[j];
      if (MODE == 1 && bias) y += b[j];
      o[j] = y;
    }
    RowCols<T>::store(out + size_t(row) * cols, cols, o);
  }
}

// A CTA per row, with the row added up in the order of norm_fwd_rows_kernel, so that its result does not depend on which of the two a call takes:
// thread t stands for threads t, t + 256, ... of a ring CTA (`ring_threads`, a multiple of 32), which own the same columns and end up in the
// same place among the warps' sums.  Several rows per SM in flight, each in registers as it lies in memory, no row waits for another's barrier; where
// the lines lie: norm_takes_row_cta.  RMSNorm bf16 4000 x 5120, input in L2 / in memory: 12.8 / 16.6 us (rings 17.0 / 17.8; converted to fp32 while it
// waits 13.5 / 17.5), 8192 x 8192 43.6 us, 6.2 TB/s (rings 51.0; converted 49.7); LayerNorm bf16 4000 x 4096 13.8 / 18.0, 8192 x 8192 56 us, 4.8 TB/s
// (rings 69).
template <typename T, int MODE, int MAXV>
__global__ void __launch_bounds__(NORM_THREADS, norm_row_ctas_per_sm<T, MODE, MAXV, false>())
norm_fwd_row_kernel(const T* __restrict__ x, const T* __restrict__ weight, const T* __restrict__ bias, T* __restrict__ out, float* __restrict__ rstd_out,
                    float* __restrict__ mean_out, int cols, int ring_threads, float eps) {
  constexpr int CHUNKS = RowCols<T>::CHUNKS, WIDTH = RowCols<T>::WIDTH;
  __shared__ float2 warp_sums[MAXV * NORM_THREADS / 32];
  pdl_wait();
  const size_t at = size_t(blockIdx.x) * cols;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto column = [&](int i, int chunk) { return (int(threadIdx.x) + i * NORM_THREADS + chunk * ring_threads) * WIDTH; };
  auto mine = [&](int i, int chunk) { return int(threadIdx.x) + i * NORM_THREADS < ring_threads && column(i, chunk) < cols; };
  auto load = [&](const T* row, int i) {
    Raw8<T> r;
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) r.u[c] = mine(i, c) ? *reinterpret_cast<const uint4*>(row + column(i, c)) : make_uint4(0, 0, 0, 0);
    return r;
  };
  constexpr bool EARLY = sizeof(T) * MAXV == 2;
  Raw8<T> held[MAXV], wr[EARLY ? MAXV : 1], br[EARLY && MODE == 1 ? MAXV : 1];
#pragma unroll
  for (int i = 0; i < MAXV; ++i) held[i] = load(x + at, i);
  if constexpr (EARLY) {
#pragma unroll
    for (int i = 0; i < MAXV; ++i) {
      if (weight) wr[i] = load(weight, i);
      if constexpr (MODE == 1) { if (bias) br[i] = load(bias, i); }
    }
  }
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    float s1 = 0.f, s2 = 0.f, v[8];
    unpack(held[i], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s1 += v[j];
      s2 += v[j] * v[j];
    }
    if (MODE == 1) s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    if (lane == 0) warp_sums[warp + i * (NORM_THREADS / 32)] = make_float2(s1, s2);
  }
  __syncthreads();
  const float2 sums = lane < ring_threads >> 5 ? warp_sums[lane] : make_float2(0.f, 0.f);
  const float s1 = MODE == 1 ? warp_sum(sums.x) : 0.f, s2 = warp_sum(sums.y);
  const float inv_n = 1.f / float(cols);
  const float mean = MODE == 1 ? s1 * inv_n : 0.f;
  const float var = MODE == 1 ? fmaxf(s2 * inv_n - mean * mean, 0.f) : s2 * inv_n;
  const float rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0) {
    if (rstd_out) rstd_out[blockIdx.x] = rstd;
    if (mean_out) mean_out[blockIdx.x] = mean;
  }
#pragma unroll
  for (int i = 0; i < MAXV; ++i) {
    float v[8], w[8], b[8], o[8];
    unpack(held[i], v);
    if (weight) unpack(EARLY ? wr[EARLY ? i : 0] : load(weight, i), w);
    if (MODE == 1 && bias) unpack(EARLY ? br[EARLY && MODE == 1 ? i : 0] : load(bias, i), b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float y = (v[j] - mean) * rstd;
      if (weight) y *= w[j];
      if (MODE == 1 && bias) y += b[j];
      o[j] = y;
    }
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      if (!mine(i, c)) continue;
      if constexpr (CHUNKS == 1) Vec8<T>::store(out + at + column(i, 0), o);
      else *reinterpret_cast<float4*>(out + at + column(i, c)) = make_float4(o[4 * c], o[4 * c + 1], o[4 * c + 2], o[4 * c + 3]);
    }
  }
}

// out[c] = sum over parts of part[p][c] (blockIdx.y: 0 = weight, 1 = bias).  32 columns x 32 rows of partials per step, so that
// every partial row's loads are independent; the summation order depends on the number of partials only.
template <typename O>
__global__ void __launch_bounds__(1024)
norm_bwd_reduce_kernel(const float* __restrict__ part_w, const float* __restrict__ part_b, O* __restrict__ dweight, O* __restrict__ dbias,
                       int parts, int cols) {
  __shared__ float tile[32][33];
  const float* part = blockIdx.y ? part_b : part_w;
  O* out = blockIdx.y ? dbias : dweight;
  if (!out) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < cols) {
#pragma unroll 4
    for (int r = ty; r < parts; r += 32) s += part[size_t(r) * cols + c];
  }
  tile[ty][tx] = s;
  __syncthreads();
  const float t = warp_sum(tile[tx][ty]);  // warp ty sums column ty of the tile
  const int co = blockIdx.x * 32 + ty;
  if (tx == 0 && co < cols) out[co] = from_f<O>(t);
}

// Column sums of bf16 rows in fp32 (the gradient of a bias): 64 columns per CTA, 32 rows side by side, a share of the rows per blockIdx.y.  With one share
// the sums are stored as they are wanted; with several they are partials for norm_bwd_reduce_kernel.  Sums run in an order that depends on the shape only.
// Bound by the one read of the rows, small ones by latency (a reduction and a cast as tensor operations in brackets, us): 100 x 3072 2.4 (5.4), 1000 x 3072
// 5.6 (20.6), 8192 x 768 8.7 (22.7), 8192 x 12288 36 (50), 32768 x 5120 53 (74).
constexpr int CS_ROWS = 32, CS_COLS = 64;
template <typename O>
__global__ void __launch_bounds__(256)
col_sum_kernel(const bf16* __restrict__ g, O* __restrict__ out, int rows, int cols, int share) {
  __shared__ float tile[CS_ROWS][CS_COLS + 4];
  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3, c = blockIdx.x * CS_COLS + tx * 8;
  const int first = blockIdx.y * share, last = min(rows, first + share);
  float s[8] = {};
  if (c < cols) {
#pragma unroll 4
    for (int r = first + ty; r < last; r += CS_ROWS) {
      float v[8];
      Vec8<bf16>::load(g + size_t(r) * cols + c, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] += v[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) tile[ty][tx * 8 + j] = s[j];
  __syncthreads();
  // four threads per column, eight rows each
  const int col = threadIdx.x >> 2, q = threadIdx.x & 3;
  float t = 0.f;
#pragma unroll
  for (int r = 0; r < CS_ROWS / 4; ++r) t += tile[q * (CS_ROWS / 4) + r][col];
  t += __shfl_xor_sync(0xffffffffu, t, 1);
  t += __shfl_xor_sync(0xffffffffu, t, 2);
  const int co = blockIdx.x * CS_COLS + col;
  if (q == 0 && co < cols) out[size_t(blockIdx.y) * cols + co] = from_f<O>(t);
}

// ------------------------------------------------------------------------------------------------
// Rotary embedding on x[tokens, heads, head_dim] (in place allowed), positions[tokens] (int64) or a
// device scalar base position (for graph-replayed decode steps): pos = base[0] + token % seq.
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void rope_kernel(const T* __restrict__ x, T* __restrict__ out, const int64_t* __restrict__ positions,
                            const int* __restrict__ base_pos, int seq, int tokens, int heads, int head_dim,
                            int rotary_dim, float log2_theta, int interleaved, int inverse, long long x_stride_tok,
                            long long out_stride_tok) {
  const int half = rotary_dim >> 1;
  const long long total = (long long)tokens * heads * half;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int p = int(i % half);
    const int h = int((i / half) % heads);
    const int t = int(i / ((long long)half * heads));
    const float pos = positions ? float(positions[t]) : float(base_pos[0] + (t % seq));
    const float inv_freq = exp2f(-log2_theta * (2.f * float(p) / float(rotary_dim)));
    float s, c;
    sincosf(pos * inv_freq, &s, &c);
    if (inverse) s = -s;
    const int ia = interleaved ? 2 * p : p;
    const int ib = interleaved ? 2 * p + 1 : p + half;
    const T* xp = x + t * x_stride_tok + (long long)h * head_dim;
    T* op = out + t * out_stride_tok + (long long)h * head_dim;
    const float a = to_f<T>(xp[ia]), b = to_f<T>(xp[ib]);
    op[ia] = from_f<T>(a * c - b * s);
    op[ib] = from_f<T>(b * c + a * s);
  }
}

// bf16 fast path with 16-byte accesses: a thread owns one chunk of a token - 8 consecutive elements of the first rotary half
// with their partners in the second (split layout), or 4 adjacent pairs (interleaved) - and walks heads hg, hg + groups, ...
// with it: the angles (exp2f and sincosf per pair) are the same for every head, and evaluating them once per thread and
// head is what bounded the kernel when it did.  Consecutive threads take consecutive chunks, then consecutive heads.
// 8192 tokens x 32 heads of 128: 49 us with angles per head, 27 us (5.0 TB/s) with angles per thread.
__global__ void __launch_bounds__(256)
rope_vec_kernel(const bf16* __restrict__ x, bf16* __restrict__ out, const int64_t* __restrict__ positions,
                const int* __restrict__ base_pos, int seq, int tokens, int heads, int groups, int head_dim, int rotary_dim,
                float log2_theta, int interleaved, int inverse, long long x_stride_tok, long long out_stride_tok) {
  const int half = rotary_dim >> 1;
  const int chunks = interleaved ? rotary_dim / 8 : half / 8;
  const int per_token = chunks * groups;
  const long long total = (long long)tokens * per_token;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = int(i / per_token);
    const int w = int(i - (long long)t * per_token);
    const int hg = w / chunks, e = (w - hg * chunks) * 8;
    const float pos = positions ? float(positions[t]) : float(base_pos[0] + (t % seq));
    const bf16* xp = x + t * x_stride_tok;
    bf16* op = out + t * out_stride_tok;
    if (!interleaved) {
      float cs[8], sn[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float inv_freq = exp2f(-log2_theta * (2.f * float(e + u) / float(rotary_dim)));
        sincosf(pos * inv_freq, &sn[u], &cs[u]);
        if (inverse) sn[u] = -sn[u];
      }
#pragma unroll 4
      for (int h = hg; h < heads; h += groups) {
        float a[8], b[8], ra[8], rb[8];
        Vec8<bf16>::load(xp + h * head_dim + e, a);
        Vec8<bf16>::load(xp + h * head_dim + e + half, b);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          ra[u] = a[u] * cs[u] - b[u] * sn[u];
          rb[u] = b[u] * cs[u] + a[u] * sn[u];
        }
        Vec8<bf16>::store(op + h * head_dim + e, ra);
        Vec8<bf16>::store(op + h * head_dim + e + half, rb);
      }
    } else {
      float cs[4], sn[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float inv_freq = exp2f(-log2_theta * (2.f * float((e >> 1) + u) / float(rotary_dim)));
        sincosf(pos * inv_freq, &sn[u], &cs[u]);
        if (inverse) sn[u] = -sn[u];
      }
#pragma unroll 4
      for (int h = hg; h < heads; h += groups) {
        float v[8], r[8];
        Vec8<bf16>::load(xp + h * head_dim + e, v);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          r[2 * u] = v[2 * u] * cs[u] - v[2 * u + 1] * sn[u];
          r[2 * u + 1] = v[2 * u + 1] * cs[u] + v[2 * u] * sn[u];
        }
        Vec8<bf16>::store(op + h * head_dim + e, r);
      }
    }
  }
}

// pass-through of the non-rotary tail when out != x
template <typename T>
__global__ void rope_tail_kernel(const T* __restrict__ x, T* __restrict__ out, int tokens, int heads, int head_dim,
                                 int rotary_dim, long long x_stride_tok, long long out_stride_tok) {
  const int tail = head_dim - rotary_dim;
  const long long total = (long long)tokens * heads * tail;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int p = int(i % tail);
    const int h = int((i / tail) % heads);
    const int t = int(i / ((long long)tail * heads));
    out[t * out_stride_tok + (long long)h * head_dim + rotary_dim + p] = x[t * x_stride_tok + (long long)h * head_dim + rotary_dim + p];
  }
}

// ------------------------------------------------------------------------------------------------
// Activations.  kind: 1 relu, 2 gelu(erf), 3 gelu(tanh), 4 silu.  Gated variants compute act(gate) * up.
// ------------------------------------------------------------------------------------------------
// act(x), and with GRAD its derivative, sharing the transcendental
template <int KIND, bool GRAD>
__device__ __forceinline__ float act_eval(float x, float& grad) {
  if (KIND == 1) {
    if (GRAD) grad = x > 0.f ? 1.f : 0.f;
    return fmaxf(x, 0.f);
  }
  if (KIND == 2) {
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    if (GRAD) grad = cdf + x * 0.3989422804014327f * expf(-0.5f * x * x);
    return x * cdf;
  }
  if (KIND == 3) {
    const float t = tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x));
    if (GRAD) grad = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * 0.7978845608028654f * (1.f + 3.f * 0.044715f * x * x);
    return 0.5f * x * (1.f + t);
  }
  if (KIND == 4) {
    const float e = 1.f + expf(-x);
    if (GRAD) {
      const float s = 1.f / e;
      grad = s * (1.f + x * (1.f - s));
    }
    return x / e;
  }
  if (GRAD) grad = 1.f;
  return x;
}

// Two 8-element vectors per thread and step (see act_grid), one instantiation per activation, no row division where rows lie one
// after another (8192 x 11008 gated, 541 MB forward and 902 MB backward: silu 134 -> 108 us and 227 -> 165 us, gelu 145 -> 113 and 321 -> 172,
// gelu(tanh) 128 -> 98 and 226 -> 148).  Memory-bound with relu (89 and 146 us); expf, erff and the IEEE divisions cost the others
// up to 24 us on top.  The hardware exponential and reciprocal would take silu to 92 and 147 us, at the cost of digits (an error of
// 1.16 |x| units in the last place).  Logical shape [rows, cols]; gate / up may be column slices of a wider fused projection
// (leading dims); DENSE: they are not, and a vector's position is its index.
template <typename T, int KIND, bool DENSE>
__global__ void __launch_bounds__(256)
act_fwd_kernel(const T* __restrict__ gate, const T* __restrict__ up, T* __restrict__ out, long long nvec, int cols, long long gate_ld, long long up_ld) {
  constexpr int U = 2;
  const int vec_per_row = cols >> 3;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < nvec; i0 += U * step) {
    Raw8<T> g[U], u[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const long long i = i0 + k * step;
      if (i < nvec) {
        const long long r = DENSE ? 0 : i / vec_per_row;
        const long long c = (DENSE ? i : i - r * vec_per_row) * 8;
        g[k] = load_raw(gate + r * gate_ld + c);
        if (up) u[k] = load_raw(up + r * up_ld + c);
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const long long i = i0 + k * step;
      if (i < nvec) {
        float gv[8], uv[8], o[8], unused;
        unpack(g[k], gv);
        if (up) unpack(u[k], uv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = act_eval<KIND, false>(gv[j], unused) * (up ? uv[j] : 1.f);
        Vec8<T>::store(out + i * 8, o);
      }
    }
  }
}

template <typename T, int KIND>
__global__ void __launch_bounds__(256)
act_bwd_kernel(const T* __restrict__ dout, const T* __restrict__ gate, const T* __restrict__ up, T* __restrict__ dgate, T* __restrict__ dup, long long nvec) {
  constexpr int U = 2;
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x; i0 < nvec; i0 += U * step) {
    Raw8<T> d[U], g[U], u[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const long long i = i0 + k * step;
      if (i < nvec) {
        d[k] = load_raw(dout + i * 8);
        g[k] = load_raw(gate + i * 8);
        if (up) u[k] = load_raw(up + i * 8);
      }
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const long long i = i0 + k * step;
      if (i < nvec) {
        float dv[8], gv[8], uv[8], dg[8], du[8];
        unpack(d[k], dv);
        unpack(g[k], gv);
        if (up) unpack(u[k], uv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float grad;
          const float f = act_eval<KIND, true>(gv[j], grad);
          dg[j] = dv[j] * grad * (up ? uv[j] : 1.f);
          du[j] = dv[j] * f;
        }
        Vec8<T>::store(dgate + i * 8, dg);
        if (up) Vec8<T>::store(dup + i * 8, du);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Embedding gather: out[t, :] = table[ids[t], :]   (cols % 8 == 0)
// ------------------------------------------------------------------------------------------------
template <typename T>
__global__ void embedding_kernel(const int64_t* __restrict__ ids, const T* __restrict__ table, T* __restrict__ out,
                                 int tokens, int cols, long long table_ld, long long out_ld) {
  pdl_wait();
  const int vec_per_row = cols >> 3;
  const long long total = (long long)tokens * vec_per_row;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int t = int(i / vec_per_row);
    const int c = int(i % vec_per_row) * 8;
    const int64_t id = ids[t];
    if constexpr (sizeof(T) == 2) {
      *reinterpret_cast<uint4*>(out + t * out_ld + c) = *reinterpret_cast<const uint4*>(table + id * table_ld + c);
    } else {
      reinterpret_cast<float4*>(out + t * out_ld + c)[0] = reinterpret_cast<const float4*>(table + id * table_ld + c)[0];
      reinterpret_cast<float4*>(out + t * out_ld + c)[1] = reinterpret_cast<const float4*>(table + id * table_ld + c)[1];
    }
  }
}

// ------------------------------------------------------------------------------------------------
// Fused AdamW: one pass over (param, grad, exp_avg, exp_avg_sq [, fp32 master]), memory-bound.
// Bias corrections are passed pre-computed; grads may be bf16 (G = bf16) or fp32.
// ------------------------------------------------------------------------------------------------
struct AdamwArgs {
  float lr, beta1, beta2, eps, weight_decay, bc1, bc2, grad_scale;
};
__device__ __forceinline__ void adamw_update(float g, float& p, float& m, float& v, const AdamwArgs& a) {
  g *= a.grad_scale;
  m = a.beta1 * m + (1.f - a.beta1) * g;
  v = a.beta2 * v + (1.f - a.beta2) * g * g;
  p *= 1.f - a.lr * a.weight_decay;
  p -= a.lr * (m / a.bc1) / (sqrtf(v / a.bc2) + a.eps);
}

// VEC: 8 elements per thread and step with 16-byte accesses (all pointers 16-byte aligned; the last n % 8 elements are done one
// by one): up to ten independent 16-byte loads per thread are in flight, where the element-wise form has five of 2 to 4 bytes
// (202 M parameters with master weights: 1260 us element-wise, 944 us = 6.4 TB/s in vectors).  A thread's eight updates are a chain
// of square roots and divisions that few threads do not hide: below ADAMW_VEC_MIN elements one thread per element is faster (bf16
// with master weights, element-wise and in vectors: 4096 elements 2.1 and 3.3 us, 100 000 2.6 and 3.6, 400 000 4.4 and 4.6,
// 600 000 5.6 and 4.8).
constexpr long long ADAMW_VEC_MIN = 1 << 19;

template <typename P, typename G, bool VEC>
__global__ void __launch_bounds__(256)
adamw_kernel(P* __restrict__ param, const G* __restrict__ grad, float* __restrict__ m, float* __restrict__ v, float* __restrict__ master,
             long long n, const AdamwArgs a) {
  const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  const long long nvec = VEC ? n >> 3 : 0;
  for (long long i = tid; i < nvec; i += step) {
    float g[8], p[8], mi[8], vi[8];
    Vec8<G>::load(grad + i * 8, g);
    Vec8<float>::load(m + i * 8, mi);
    Vec8<float>::load(v + i * 8, vi);
    if (master) Vec8<float>::load(master + i * 8, p);
    else Vec8<P>::load(param + i * 8, p);
#pragma unroll
    for (int j = 0; j < 8; ++j) adamw_update(g[j], p[j], mi[j], vi[j], a);
    Vec8<float>::store(m + i * 8, mi);
    Vec8<float>::store(v + i * 8, vi);
    if (master) Vec8<float>::store(master + i * 8, p);
    Vec8<P>::store(param + i * 8, p);
  }
  for (long long i = nvec * 8 + tid; i < n; i += step) {
    float p = master ? master[i] : to_f<P>(param[i]), mi = m[i], vi = v[i];
    adamw_update(to_f<G>(grad[i]), p, mi, vi, a);
    m[i] = mi;
    v[i] = vi;
    if (master) master[i] = p;
    param[i] = from_f<P>(p);
  }
}

template <typename A, typename B>
__global__ void cast_kernel(const A* __restrict__ in, B* __restrict__ out, long long n, float scale) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = from_f<B>(to_f<A>(in[i]) * scale);
}

static inline int grid_for(long long work, int threads) {
  long long g = (work + threads - 1) / threads;
  if (g > 148LL * 16) g = 148LL * 16;
  if (g < 1) g = 1;
  return int(g);
}

// The activation kernels take two vectors per thread where the chip is full; below 2^18 vectors (all threads resident at once) a
// thread takes one, so that the chain of one thread is half as long (gated silu, two per thread and one: 100 x 768 2.8 and 2.4 us
// forward, 3.6 and 2.6 us backward; 700 x 2048 3.7 and 3.4, 5.0 and 4.8; relu of 1000 x 3072 3.0 and 3.4).
static inline int act_grid(long long nvec) { return grid_for(nvec < (1 << 18) ? nvec : (nvec + 1) / 2, 256); }

}  // namespace tpb

using namespace tpb;

#define TPB_CHECK_LAUNCH() return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA

// Threads of a CTA whose threads own 8 columns each, and CTAs of them that fill an SM, up to 16.
static inline int norm_row_threads(int cols) { return (cols / 8 + 31) / 32 * 32; }
static inline int norm_row_ctas(int rows, int cols, int threads_per_sm) {
  const int per_sm = threads_per_sm / norm_row_threads(cols);
  const int ctas = 148 * (per_sm > 16 ? 16 : (per_sm < 1 ? 1 : per_sm));
  return rows < ctas ? rows : ctas;
}

// Widths whose rows (nearly) fill 256 threads with one or two vectors each.
static inline bool norm_filled(int cols) { return (cols > NORM_THREADS * 6 && cols <= NORM_THREADS * 8) || (cols > NORM_THREADS * 12 && cols <= NORM_THREADS * 16); }

// norm_fwd_row_kernel (true) or norm_fwd_rows_kernel for a forward without a residual, which give the same bits.  Times in us as row / ring, "hot"
// with the input in L2, as the kernel before leaves it, "cold" with it in memory.
static inline bool norm_takes_row_cta(int rows, int cols, int mode, int dtype) {
  // fp32: RMSNorm of many rows that fill the threads (8192 x 4096 42.1 / 47.3, 16384 x 2048 41.4 / 47.8; cold 4000 x 2048 12.6 / 12.3, 2000 x 4096 12.7 / 12.5)
  if (dtype == 1) return mode == 0 && norm_filled(cols) && rows >= 8192;
  // one row per SM: the ring kernel's CTA has more threads for it (LayerNorm 100 x 8192 4.2 / 3.3, 20 x 5120 3.5 / 2.6; RMSNorm 100 x 8192 3.4 / 3.0)
  if (cols > 1536 && rows <= 148) return false;
  // wide rows: RMSNorm 2000 x 5120 hot 7.2 / 9.5, cold 10.1 / 10.7; 2000 x 3072 5.7 / 7.3, 7.5 / 7.7; LayerNorm 2000 x 5120 10.6 / 11.9, 13.3 / 13.8; 1000 x
  // 8192 9.0 / 11.2, 11.3 / 12.8.  But 4000 x 2560 9.3 / 10.0, 11.8 / 10.7, LayerNorm 4000 x 3072 13.2 / 13.5, 16.6 / 16.1: rings
  if (cols > 3072 || (mode == 0 && cols > 2560)) return true;
  // middle widths: hot faster, cold slower (RMSNorm 4000 x 1536 6.5 / 7.0, 8.6 / 7.6; LayerNorm 4000 x 2048 8.9 / 10.1, 10.8 / 11.0), so by whether
  // input and output can be hot
  if (mode == 0 ? cols > 1024 && cols <= 1536 : cols > 1536 && cols <= 2048) return (long long)rows * cols <= 1 << 24;
  // narrow RMSNorm rows that are all resident at once (300 x 768 2.2 / 2.3, 1000 x 1024 2.8 / 2.8; 2000 x 768 3.9 / 3.2, 300 x 256 2.1 / 2.0)
  return mode == 0 && cols > 256 && cols <= 1024 && rows <= 8 * 148;
}

// Lets a kernel have a ring of the widest row (1024 threads: 192 KB), once per device.
template <auto KERNEL>
static bool norm_ring_allowed() {
  static std::atomic<bool> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (!done[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, 192 * 1024) != cudaSuccess) return false;
    done[dev].store(true, std::memory_order_release);
  }
  return true;
}

// dtype: 0 = bf16, 1 = fp32.  mode: 0 = RMSNorm, 1 = LayerNorm.
extern "C" int tpb_norm_fwd(const void* x, const void* residual, const void* weight, const void* bias, void* out,
                            void* sum_out, float* rstd_out, float* mean_out, int rows, int cols, float eps, int mode,
                            int dtype, void* stream_) {
  if (!x || !out || rows <= 0 || cols <= 0) return TPB_ERR_ARG;
  if ((cols & 7) || cols > NORM_THREADS * 8 * NORM_MAXV) return TPB_ERR_SIZE;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  // bf16 RMSNorm rows that fill 256 threads: a CTA per row in an order of its own whatever their number (600 x 4096 3.0 us, ring 4.4; 1000 x 2048 3.0
  // and 3.7; 20 x 4096 2.1 and 2.4; 2000 x 4096 in memory 7.9 and 9.3)
  const bool one_cta = mode == 0 && norm_filled(cols) && dtype == 0;
  if (!residual && !one_cta && cols <= NORM_BWD_MAXC && norm_takes_row_cta(rows, cols, mode, dtype)) {
#define LAUNCH(T, M, V)                                                                                                                        \
  launch_kernel(norm_fwd_row_kernel<T, M, V>, dim3(rows), dim3(NORM_THREADS), 0, s, (const T*)x, (const T*)weight, (const T*)bias, (T*)out, rstd_out, \
                mean_out, cols, norm_row_threads(cols), eps)
#define LAUNCH_V(T, M)                                                                                                  \
  do {                                                                                                                  \
    if (cols <= NORM_THREADS * 8) LAUNCH(T, M, 1);                                                                      \
    else if (cols <= NORM_THREADS * 16) LAUNCH(T, M, 2);                                                                \
    else if constexpr (sizeof(T) == 2) { if (cols <= NORM_THREADS * 24) LAUNCH(T, M, 3); else LAUNCH(T, M, 4); }        \
  } while (0)
    if (dtype == 1) LAUNCH_V(float, 0);
    else if (mode) LAUNCH_V(bf16, 1);
    else LAUNCH_V(bf16, 0);
#undef LAUNCH_V
#undef LAUNCH
    TPB_CHECK_LAUNCH();
  }
  if (!residual && cols <= NORM_BWD_MAXC && !one_cta) {
    const int threads = norm_row_threads(cols);
    const dim3 grid(norm_row_ctas(rows, cols, dtype == 0 ? 2048 : 1024));
#define LAUNCH(T, M)                                                                                                                \
  do {                                                                                                                              \
    if (!norm_ring_allowed<norm_fwd_rows_kernel<T, M>>()) return TPB_ERR_CUDA;                                                      \
    launch_kernel(norm_fwd_rows_kernel<T, M>, grid, dim3(threads), RowRing<T, 1>::bytes(threads), s, (const T*)x, (const T*)weight, \
                  (const T*)bias, (T*)out, rstd_out, mean_out, unsigned(rows), cols, eps);                                          \
  } while (0)
    if (dtype == 0) { if (mode) LAUNCH(bf16, 1); else LAUNCH(bf16, 0); }
    else            { if (mode) LAUNCH(float, 1); else LAUNCH(float, 0); }
#undef LAUNCH
    TPB_CHECK_LAUNCH();
  }
  // (without a residual only rows wider than the rings' and the bf16 RMSNorm rows above come here)
#define LAUNCH3(T, M, V)                                                                                                                     \
  do {                                                                                                                                       \
    auto kernel = norm_fwd_kernel<T, M, V, true>;                                                                                            \
    if constexpr (V == 8 || (M == 0 && sizeof(T) == 2 && V <= 2)) { if (!residual) kernel = norm_fwd_kernel<T, M, V, false>; }               \
    launch_kernel(kernel, dim3(rows), dim3(NORM_THREADS), 0, s, (const T*)x, (const T*)residual, (const T*)weight, (const T*)bias, (T*)out,  \
                  (T*)sum_out, rstd_out, mean_out, cols, eps);                                                                               \
  } while (0)
#define LAUNCH(T, M)                                                                     \
  do {                                                                                   \
    if (cols <= NORM_THREADS * 8) LAUNCH3(T, M, 1);                                      \
    else if (cols <= NORM_THREADS * 16) LAUNCH3(T, M, 2);                                \
    else if (cols <= NORM_THREADS * 32) LAUNCH3(T, M, 4);                                \
    else LAUNCH3(T, M, 8);                                                               \
  } while (0)
  if (dtype == 0) { if (mode) LAUNCH(bf16, 1); else LAUNCH(bf16, 0); }
  else            { if (mode) LAUNCH(float, 1); else LAUNCH(float, 0); }
#undef LAUNCH
#undef LAUNCH3
  TPB_CHECK_LAUNCH();
}

// Rows of fp32 partials that tpb_norm_bwd needs (= its CTAs): part_w / part_b hold that many rows of `cols` floats.  (More than 16
// CTAs of narrow rows per SM: more partials would cost more than their CTAs bring.)
extern "C" int tpb_norm_bwd_parts(int rows, int cols) { return norm_row_ctas(rows, cols, 1024); }

// dweight / dbias (either may be null, with its partials) are written, not accumulated; grad_dtype: 0 = bf16, 1 = fp32.
extern "C" int tpb_norm_bwd(const void* dy, const void* x, const void* weight, const float* rstd, const float* mean,
                            void* dx, float* part_w, float* part_b, void* dweight, void* dbias, int rows, int cols, int mode, int dtype,
                            int grad_dtype, void* stream_) {
  if (!dy || !x || !dx || !rstd || rows <= 0 || cols <= 0 || (mode && !mean) || (dweight && !part_w) || (dbias && (!part_b || !mode))) return TPB_ERR_ARG;
  if ((cols & 7) || cols > NORM_BWD_MAXC) return TPB_ERR_SIZE;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const int grid = norm_row_ctas(rows, cols, 1024), threads = norm_row_threads(cols);
  if (!dweight) part_w = nullptr;
  if (!dbias) part_b = nullptr;
#define LAUNCH(T, M)                                                                                                                    \
  do {                                                                                                                                 \
    const size_t ring = RowRing<T, 2>::bytes(threads);                                                                                 \
    if (!norm_ring_allowed<norm_bwd_kernel<T, M>>()) return TPB_ERR_CUDA;                                                                \
    norm_bwd_kernel<T, M><<<grid, threads, ring, s>>>((const T*)dy, (const T*)x, (const T*)weight, rstd, mean, (T*)dx, part_w, part_b, \
                                                      rows, cols);                                                                     \
  } while (0)
  if (dtype == 0) { if (mode) LAUNCH(bf16, 1); else LAUNCH(bf16, 0); }
  else            { if (mode) LAUNCH(float, 1); else LAUNCH(float, 0); }
#undef LAUNCH
  if (dweight || dbias) {
    const dim3 rgrid((cols + 31) / 32, dbias ? 2 : 1);
    if (grad_dtype == 0)
      norm_bwd_reduce_kernel<bf16><<<rgrid, 1024, 0, s>>>(part_w, part_b, (bf16*)dweight, (bf16*)dbias, grid, cols);
    else
      norm_bwd_reduce_kernel<float><<<rgrid, 1024, 0, s>>>(part_w, part_b, (float*)dweight, (float*)dbias, grid, cols);
  }
  TPB_CHECK_LAUNCH();
}

// Shares of the rows that tpb_col_sum works on side by side (fp32 partials [shares][cols] that it needs where there are several): as many as give six
// CTAs per SM, of 64 rows at least.
extern "C" int tpb_col_sum_parts(int rows, int cols) {
  const int column_ctas = (cols + tpb::CS_COLS - 1) / tpb::CS_COLS, most = (rows + 63) / 64, wanted = (6 * 148 + column_ctas - 1) / column_ctas;
  return rows <= 256 ? 1 : most < wanted ? most : wanted;
}

// out[c] = sum over the rows of g[rows, cols] (bf16, contiguous, 16-byte aligned, cols a multiple of 8) in fp32; out_dtype: 0 = bf16, 1 = fp32.
extern "C" int tpb_col_sum(const void* g, void* out, float* partials, int rows, int cols, int out_dtype, void* stream_) {
  if (!g || !out || rows <= 0 || cols <= 0) return TPB_ERR_ARG;
  if ((cols & 7) || (reinterpret_cast<uintptr_t>(g) & 15)) return TPB_ERR_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const int parts = tpb_col_sum_parts(rows, cols), share = (rows + parts - 1) / parts;
  if (parts > 1 && !partials) return TPB_ERR_ARG;
  const dim3 grid((cols + CS_COLS - 1) / CS_COLS, parts), rgrid((cols + 31) / 32);
  if (parts > 1 || out_dtype) col_sum_kernel<float><<<grid, 256, 0, s>>>((const bf16*)g, parts > 1 ? partials : (float*)out, rows, cols, share);
  else col_sum_kernel<bf16><<<grid, 256, 0, s>>>((const bf16*)g, (bf16*)out, rows, cols, share);
  if (parts > 1) {
    if (out_dtype) norm_bwd_reduce_kernel<float><<<rgrid, 1024, 0, s>>>(partials, nullptr, (float*)out, nullptr, parts, cols);
    else norm_bwd_reduce_kernel<bf16><<<rgrid, 1024, 0, s>>>(partials, nullptr, (bf16*)out, nullptr, parts, cols);
  }
  TPB_CHECK_LAUNCH();
}

// Head groups of the rotary kernels: threads per (token, chunk).  Each thread reuses its angles for heads / groups heads, up to
// 8, as long as that leaves 512 threads per SM (below that the launch is latency-bound and more threads beat fewer angles).
extern "C" int tpb_rope_head_groups(long long token_chunks, int heads) {
  int per_thread = 8;
  while (per_thread > 1 && token_chunks * ((heads + per_thread - 1) / per_thread) < 148LL * 512) per_thread >>= 1;
  return (heads + per_thread - 1) / per_thread;
}

extern "C" int tpb_rope(const void* x, void* out, const int64_t* positions, const int* base_pos, int seq, int tokens,
                        int heads, int head_dim, int rotary_dim, float theta, int interleaved, int inverse,
                        long long x_stride_tok, long long out_stride_tok, int dtype, void* stream_) {
  if (!x || !out || (!positions && !base_pos) || tokens <= 0 || (rotary_dim & 1) || rotary_dim > head_dim) return TPB_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const long long work = (long long)tokens * heads * (rotary_dim / 2);
  const float l2t = log2f(theta);
  const int half_ = rotary_dim / 2;
  const bool vec_ok = dtype == 0 && head_dim % 8 == 0 && (interleaved ? rotary_dim % 8 == 0 : half_ % 8 == 0) && rotary_dim > 0 &&
                      !(x_stride_tok & 7) && !(out_stride_tok & 7) && !((uintptr_t)x & 15) && !((uintptr_t)out & 15);
  if (vec_ok) {
    const int chunks = interleaved ? rotary_dim / 8 : half_ / 8;
    const int groups = tpb_rope_head_groups((long long)tokens * chunks, heads);
    rope_vec_kernel<<<grid_for((long long)tokens * chunks * groups, 256), 256, 0, s>>>((const bf16*)x, (bf16*)out, positions, base_pos, seq, tokens,
                                                                                       heads, groups, head_dim, rotary_dim, l2t, interleaved,
                                                                                       inverse, x_stride_tok, out_stride_tok);
  } else if (dtype == 0)
    rope_kernel<bf16><<<grid_for(work, 256), 256, 0, s>>>((const bf16*)x, (bf16*)out, positions, base_pos, seq, tokens, heads,
                                                          head_dim, rotary_dim, l2t, interleaved, inverse, x_stride_tok, out_stride_tok);
  else
    rope_kernel<float><<<grid_for(work, 256), 256, 0, s>>>((const float*)x, (float*)out, positions, base_pos, seq, tokens, heads,
                                                           head_dim, rotary_dim, l2t, interleaved, inverse, x_stride_tok, out_stride_tok);
  if (x != out && rotary_dim < head_dim) {
    const long long tw = (long long)tokens * heads * (head_dim - rotary_dim);
    if (dtype == 0)
      rope_tail_kernel<bf16><<<grid_for(tw, 256), 256, 0, s>>>((const bf16*)x, (bf16*)out, tokens, heads, head_dim, rotary_dim, x_stride_tok, out_stride_tok);
    else
      rope_tail_kernel<float><<<grid_for(tw, 256), 256, 0, s>>>((const float*)x, (float*)out, tokens, heads, head_dim, rotary_dim, x_stride_tok, out_stride_tok);
  }
  TPB_CHECK_LAUNCH();
}

extern "C" int tpb_act_fwd(const void* gate, const void* up, void* out, long long rows, int cols, long long gate_ld,
                           long long up_ld, int kind, int dtype, void* stream_) {
  if (!gate || !out || rows <= 0 || cols <= 0) return TPB_ERR_ARG;
  if ((cols & 7) || (gate_ld & 7) || (up_ld & 7)) return TPB_ERR_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const long long nvec = rows * (cols / 8);
  const bool dense = (gate_ld == cols || rows == 1) && (!up || up_ld == cols || rows == 1);
#define LAUNCH2(T, K)                                                                                                                                   \
  do {                                                                                                                                                  \
    if (dense) act_fwd_kernel<T, K, true><<<act_grid(nvec), 256, 0, s>>>((const T*)gate, (const T*)up, (T*)out, nvec, cols, gate_ld, up_ld);   \
    else act_fwd_kernel<T, K, false><<<act_grid(nvec), 256, 0, s>>>((const T*)gate, (const T*)up, (T*)out, nvec, cols, gate_ld, up_ld);        \
  } while (0)
#define LAUNCH(T)                                                                                                           \
  do {                                                                                                                      \
    if (kind == 1) LAUNCH2(T, 1); else if (kind == 2) LAUNCH2(T, 2); else if (kind == 3) LAUNCH2(T, 3);                       \
    else if (kind == 4) LAUNCH2(T, 4); else LAUNCH2(T, 0);                                                                    \
  } while (0)
  if (dtype == 0) LAUNCH(bf16);
  else LAUNCH(float);
#undef LAUNCH
#undef LAUNCH2
  TPB_CHECK_LAUNCH();
}

extern "C" int tpb_act_bwd(const void* dout, const void* gate, const void* up, void* dgate, void* dup, long long n,
                           int kind, int dtype, void* stream_) {
  if (!dout || !gate || !dgate || n <= 0) return TPB_ERR_ARG;
  if (n & 7) return TPB_ERR_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const long long nvec = n / 8;
#define LAUNCH2(T, K) \
  act_bwd_kernel<T, K><<<act_grid(nvec), 256, 0, s>>>((const T*)dout, (const T*)gate, (const T*)up, (T*)dgate, (T*)dup, nvec)
#define LAUNCH(T)                                                                                                           \
  do {                                                                                                                      \
    if (kind == 1) LAUNCH2(T, 1); else if (kind == 2) LAUNCH2(T, 2); else if (kind == 3) LAUNCH2(T, 3);                       \
    else if (kind == 4) LAUNCH2(T, 4); else LAUNCH2(T, 0);                                                                    \
  } while (0)
  if (dtype == 0) LAUNCH(bf16);
  else LAUNCH(float);
#undef LAUNCH
#undef LAUNCH2
  TPB_CHECK_LAUNCH();
}

extern "C" int tpb_embedding(const int64_t* ids, const void* table, void* out, int tokens, int cols, long long table_ld,
                             long long out_ld, int dtype, void* stream_) {
  if (!ids || !table || !out || tokens <= 0) return TPB_ERR_ARG;
  if ((cols & 7) || (table_ld & 7) || (out_ld & 7)) return TPB_ERR_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const long long work = (long long)tokens * (cols / 8);
  if (dtype == 0)
    launch_kernel(embedding_kernel<bf16>, dim3(grid_for(work, 256)), dim3(256), 0, s, ids, (const bf16*)table, (bf16*)out, tokens, cols, table_ld, out_ld);
  else
    embedding_kernel<float><<<grid_for(work, 256), 256, 0, s>>>(ids, (const float*)table, (float*)out, tokens, cols, table_ld, out_ld);
  TPB_CHECK_LAUNCH();
}

extern "C" int tpb_adamw(void* param, const void* grad, float* m, float* v, float* master, long long n, float lr,
                         float beta1, float beta2, float eps, float weight_decay, int step, float grad_scale,
                         int param_dtype, int grad_is_fp32, void* stream_) {
  if (!param || !grad || !m || !v || n <= 0 || step < 1) return TPB_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const AdamwArgs a = {lr, beta1, beta2, eps, weight_decay, 1.f - powf(beta1, float(step)), 1.f - powf(beta2, float(step)), grad_scale};
  const bool vec = n >= ADAMW_VEC_MIN && !((reinterpret_cast<uintptr_t>(param) | reinterpret_cast<uintptr_t>(grad) | reinterpret_cast<uintptr_t>(m) |
                      reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(master)) & 15);
#define LAUNCH(P, G)                                                                                                                  \
  do {                                                                                                                                \
    if (vec) adamw_kernel<P, G, true><<<grid_for((n + 7) / 8, 256), 256, 0, s>>>((P*)param, (const G*)grad, m, v, master, n, a);      \
    else adamw_kernel<P, G, false><<<grid_for(n, 256), 256, 0, s>>>((P*)param, (const G*)grad, m, v, master, n, a);                   \
  } while (0)
  if (param_dtype == 0) { if (grad_is_fp32) LAUNCH(bf16, float); else LAUNCH(bf16, bf16); }
  else                  { if (grad_is_fp32) LAUNCH(float, float); else LAUNCH(float, bf16); }
#undef LAUNCH
  TPB_CHECK_LAUNCH();
}

// direction: 0 = bf16 -> fp32, 1 = fp32 -> bf16
extern "C" int tpb_cast(const void* in, void* out, long long n, float scale, int direction, void* stream_) {
  if (!in || !out || n <= 0) return TPB_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  if (direction == 0)
    cast_kernel<bf16, float><<<grid_for(n, 256), 256, 0, s>>>((const bf16*)in, (float*)out, n, scale);
  else
    cast_kernel<float, bf16><<<grid_for(n, 256), 256, 0, s>>>((const float*)in, (bf16*)out, n, scale);
  TPB_CHECK_LAUNCH();
}

// ------------------------------------------------------------------------------------------------
// bf16 matrix transpose out[c, r] = in[r, c] through a padded 64x64 shared tile (both sides coalesced)
// ------------------------------------------------------------------------------------------------
namespace tpb {
__global__ void transpose_bf16_kernel(const bf16* __restrict__ in, bf16* __restrict__ out, int rows, int cols,
                                      long long in_ld, long long out_ld) {
  __shared__ bf16 tile[64][66];
  const int r0 = blockIdx.y * 64, c0 = blockIdx.x * 64;
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    const int r = r0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      const int c = c0 + j;
      if (r < rows && c < cols) tile[i][j] = in[(long long)r * in_ld + c];
    }
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 64; i += blockDim.y) {
    const int c = c0 + i;
    for (int j = threadIdx.x; j < 64; j += blockDim.x) {
      const int r = r0 + j;
      if (r < rows && c < cols) out[(long long)c * out_ld + r] = tile[j][i];
    }
  }
}
}  // namespace tpb

extern "C" int tpb_transpose_bf16(const void* in, void* out, int rows, int cols, long long in_ld, long long out_ld,
                                  void* stream_) {
  if (!in || !out || rows <= 0 || cols <= 0) return TPB_ERR_ARG;
  dim3 grid((cols + 63) / 64, (rows + 63) / 64), block(64, 8);
  tpb::transpose_bf16_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream_)>>>(
      static_cast<const tpb::bf16*>(in), static_cast<tpb::bf16*>(out), rows, cols, in_ld, out_ld);
  TPB_CHECK_LAUNCH();
}

// ------------------------------------------------------------------------------------------------
// End of a greedy decode step in one launch: ids[b] = next_ids[b] = argmax of logits row b (the first one of equal values, a NaN
// above everything, like torch.argmax), pos[0] += 1.  One CTA per row; a row of 32000 logits is 64 KB, so the time is launch
// latency plus about one microsecond - as separate cast, argmax, copy and add kernels it was four launches.
// ------------------------------------------------------------------------------------------------
namespace tpb {
constexpr int PICK_THREADS = 512;
struct Best { float v; int i; };
__device__ __forceinline__ bool beats(const Best& a, const Best& b) {  // a comes before b in the order of torch.argmax
  const bool an = a.v != a.v, bn = b.v != b.v;
  if (an != bn) return an;
  if (an || a.v == b.v) return a.i < b.i;
  return a.v > b.v;
}
__global__ void __launch_bounds__(PICK_THREADS)
greedy_pick_kernel(const bf16* logits, long long ld, int cols, int64_t* __restrict__ next_ids, int64_t* __restrict__ ids,
                   int* __restrict__ pos) {
  __shared__ Best red[PICK_THREADS / 32];
  pdl_wait();
  const bf16* x = logits + blockIdx.x * ld;
  const int head = min(cols, int((16 - (reinterpret_cast<uintptr_t>(x) & 15)) & 15) / 2), tail = head + (cols - head) / 8 * 8;
  Best best = {-INFINITY, cols};  // (loses against every element)
#pragma unroll 4
  for (int c = head + int(threadIdx.x) * 8; c < tail; c += PICK_THREADS * 8) {
    float v[8];
    unpack(Raw8<bf16>{{ld_after_wait_v4(x + c)}}, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const Best cand = {v[j], c + j};
      if (beats(cand, best)) best = cand;
    }
  }
  const int edge = head + cols - tail;  // at most 14 elements outside the 16-byte vectors
  if (int(threadIdx.x) < edge) {
    const int c = int(threadIdx.x) < head ? int(threadIdx.x) : tail + int(threadIdx.x) - head;
    const Best cand = {bf16_bits_to_float(ld_after_wait_u16(x + c)), c};
    if (beats(cand, best)) best = cand;
  }
  auto merge = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const Best other = {__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      if (beats(other, best)) best = other;
    }
  };
  merge();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x < 32) {
    best = threadIdx.x < PICK_THREADS / 32 ? red[threadIdx.x] : Best{-INFINITY, cols};
    merge();
    if (threadIdx.x == 0) {
      next_ids[blockIdx.x] = best.i;
      ids[blockIdx.x] = best.i;
      if (blockIdx.x == 0) pos[0] += 1;
    }
  }
}
}  // namespace tpb

// early: launch as a programmatic dependent (the kernel reads nothing before the previous kernel of the stream is complete).
extern "C" int tpb_greedy_pick(const void* logits, long long ld, int rows, int cols, int64_t* next_ids, int64_t* ids, int* pos, int early, void* stream_) {
  if (!logits || !next_ids || !ids || !pos || rows <= 0 || cols <= 0 || ld < cols) return TPB_ERR_ARG;
  return launch_dependent(tpb::greedy_pick_kernel, dim3(rows), dim3(tpb::PICK_THREADS), 0, static_cast<cudaStream_t>(stream_), early != 0 || pdl_enabled(),
                          static_cast<const tpb::bf16*>(logits), ld, cols, next_ids, ids, pos) == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}
