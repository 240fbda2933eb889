// Vocab-parallel cross-entropy: each rank holds logits for its slice of the vocabulary only.
//   tpb_ce_stats : per row -> (local max, local sum of exp(logit - local max), target logit or 0) + "target is mine" flag
//   tpb_ce_loss  : the ranks' statistics -> log-sum-exp per row, mean loss over the rows whose label is not ignored, their number
//   tpb_ce_grad  : given the global log-sum-exp per row, overwrite the local logits with
//                  d loss / d logit = (softmax - onehot) * scale   (rows with an ignored label become 0)
// Only [rows, 4] floats per rank have to cross the interconnect; full logits never exist anywhere.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "tpb_api.h"

namespace tpb {

typedef __nv_bfloat16 bf16;
constexpr int CE_THREADS = 256;

__device__ __forceinline__ float ce_warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float ce_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One CTA per row, 16-byte accesses.  A row starts at any element when the pitch is odd (a vocabulary that is no multiple of 8):
// [0, head) and [tail, cols) are handled one by one, [head, tail) is 16-byte aligned.
// U vectors in flight per thread, or U = 0: every element is its own access.  Long rows hide their latency with four (8192 x 32000, 1
// and 4: statistics 130 and 117 us, gradient 174 and 162 us; 65 x 32000 8.0 and 5.8, 7.0 and 5.5 us).  Below 8192 columns a thread has
// no four vectors and their registers only cost CTAs per SM (8192 x 4000, 1 and 4: 24.8 and 29.0, 21.8 and 22.6 us; 8192 x 1000: 14.5 and
// 22.4, 9.7 and 12.3 us), below 256 most threads have none (1000 x 131, 0 and 1: 3.0 and 3.6, 2.4 and 3.2 us).  Element-wise accesses and
// two passes took 178 and 239 us for 8192 x 32000, 30 and 27 us for 8192 x 4000.
#define CE_DISPATCH(cols, LAUNCH) \
  do {                            \
    if (cols >= 8192) LAUNCH(4);  \
    else if (cols >= 256) LAUNCH(1); \
    else LAUNCH(0);               \
  } while (0)
struct CeSpan { int head, tail; };
__device__ __forceinline__ CeSpan ce_span(const bf16* x, int cols) {
  const int head = min(cols, int((16 - (reinterpret_cast<uintptr_t>(x) & 15)) & 15) / 2);
  return {head, head + (cols - head) / 8 * 8};
}
__device__ __forceinline__ void ce_unpack(const uint4& u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

// One pass over the row: every thread keeps a running maximum and the sum of exp(x - maximum), rescaled when the maximum of a
// group of loaded values exceeds it; the threads' pairs are merged at the end.
template <int U>
__global__ void __launch_bounds__(CE_THREADS)
ce_stats_kernel(const bf16* __restrict__ logits, const int64_t* __restrict__ labels, float* __restrict__ stats, int cols,
                long long ld, int vocab_start, int ignore_index) {
  const long long row = blockIdx.x;
  const bf16* x = logits + row * ld;
  __shared__ float red_m[CE_THREADS / 32], red_s[CE_THREADS / 32];
  const CeSpan span = U ? ce_span(x, cols) : CeSpan{cols, cols};
  float m = -INFINITY, s = 0.f;
  auto raise = [&](float group_max) {  // exp(-inf - -inf) must not arise while nothing finite has been seen
    if (group_max > m) {
      s *= expf(m - group_max);
      m = group_max;
    }
    return m == -INFINITY ? 0.f : m;
  };
  if constexpr (U > 0)
    for (int c = span.head + threadIdx.x * 8; c < span.tail; c += U * CE_THREADS * 8) {
    uint4 raw[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int ck = c + k * CE_THREADS * 8;
      raw[k] = ck < span.tail ? *reinterpret_cast<const uint4*>(x + ck) : make_uint4(0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u, 0xFF80FF80u);  // -inf
    }
    float v[U][8], gm = -INFINITY;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      ce_unpack(raw[k], v[k]);
#pragma unroll
      for (int j = 0; j < 8; ++j) gm = fmaxf(gm, v[k][j]);
    }
    const float base = raise(gm);
#pragma unroll
    for (int k = 0; k < U; ++k) {
      float part = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) part += expf(v[k][j] - base);
      s += part;
    }
  }
  const int edge = span.head + cols - span.tail;  // outside the vectors: at most 14 elements, or the whole row (U = 0)
  for (int i = threadIdx.x; i < edge; i += CE_THREADS) {
    const float v = __bfloat162float(x[i < span.head ? i : span.tail + i - span.head]);
    const float base = raise(v);
    s += expf(v - base);
  }
  // merge (maximum, sum) over the CTA; a pair without a finite maximum carries no mass (or a NaN that has to survive)
  const float wm = ce_warp_max(m);
  s = ce_warp_sum(m == wm ? s : s * expf(m - wm));
  if ((threadIdx.x & 31) == 0) {
    red_m[threadIdx.x >> 5] = wm;
    red_s[threadIdx.x >> 5] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mm = red_m[0], t = 0.f;
    for (int w = 1; w < CE_THREADS / 32; ++w) mm = fmaxf(mm, red_m[w]);
    for (int w = 0; w < CE_THREADS / 32; ++w) t += red_m[w] == mm ? red_s[w] : red_s[w] * expf(red_m[w] - mm);
    if (mm == -INFINITY) t = NAN;  // no finite logit in this slice: exp(-inf - -inf)
    const long long label = labels[row];
    const long long local = label - vocab_start;
    const bool mine = label != ignore_index && local >= 0 && local < cols;
    stats[row * 4 + 0] = mm;
    stats[row * 4 + 1] = t;
    stats[row * 4 + 2] = mine ? __bfloat162float(x[local]) : 0.f;
    stats[row * 4 + 3] = mine ? 1.f : 0.f;
  }
}

// Sums over the CTA, in a fixed order.
__device__ __forceinline__ void ce_block_sum(float& a, int& n) {
  __shared__ float red_a[CE_THREADS / 32];
  __shared__ int red_n[CE_THREADS / 32];
  a = ce_warp_sum(a);
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) {
    red_a[threadIdx.x >> 5] = a;
    red_n[threadIdx.x >> 5] = n;
  }
  __syncthreads();
  a = 0.f;
  n = 0;
#pragma unroll
  for (int w = 0; w < CE_THREADS / 32; ++w) {
    a += red_a[w];
    n += red_n[w];
  }
}

// One thread per row; the CTA's share of the loss and of the count goes into one partial, which ce_mean_kernel adds up in a fixed
// order.  A handful of bytes per row: what counts are the launches.  As a dozen PyTorch operators this step kept the GPU busy for 45 us
// (head of 8192 x 32000 x 4096 with its loss, forward and backward: 5393 -> 5335 us with these two kernels).
__global__ void __launch_bounds__(CE_THREADS)
ce_loss_kernel(const float4* __restrict__ stats, const int64_t* __restrict__ labels, float* __restrict__ lse, float2* __restrict__ partials, int world,
               int rows, int ignore_index) {
  const int row = blockIdx.x * CE_THREADS + threadIdx.x;
  float share = 0.f;
  int counts = 0;
  if (row < rows) {
    float gmax = -INFINITY, sum = 0.f, target = 0.f;
    for (int r = 0; r < world; ++r) gmax = fmaxf(gmax, stats[(long long)r * rows + row].x);
    for (int r = 0; r < world; ++r) {
      const float4 st = stats[(long long)r * rows + row];
      sum += st.y * expf(st.x - gmax);
      target += st.z;
    }
    const float l = gmax + logf(sum);
    lse[row] = l;
    counts = labels[row] != ignore_index;
    share = (l - target) * float(counts);  // (a product: what is not finite stays visible in an ignored row too)
  }
  ce_block_sum(share, counts);
  if (threadIdx.x == 0) partials[blockIdx.x] = make_float2(share, __int_as_float(counts));
}

__global__ void __launch_bounds__(CE_THREADS)
ce_mean_kernel(const float2* __restrict__ partials, int count, float* __restrict__ loss, float* __restrict__ n_valid) {
  float a = 0.f;
  int n = 0;
  for (int i = threadIdx.x; i < count; i += CE_THREADS) {
    const float2 v = partials[i];
    a += v.x;
    n += __float_as_int(v.y);
  }
  ce_block_sum(a, n);
  if (threadIdx.x == 0) {
    n_valid[0] = float(max(n, 1));
    loss[0] = a / n_valid[0];
  }
}

template <int U>
__global__ void __launch_bounds__(CE_THREADS)
ce_grad_kernel(bf16* __restrict__ logits, const int64_t* __restrict__ labels, const float* __restrict__ lse, int cols,
               long long ld, int vocab_start, int ignore_index, const float* __restrict__ scale_ptr) {
  const long long row = blockIdx.x;
  bf16* x = logits + row * ld;
  const CeSpan span = U ? ce_span(x, cols) : CeSpan{cols, cols};
  const long long label = labels[row];
  const int edge = span.head + cols - span.tail;
  if (label == ignore_index) {
    for (int c = span.head + threadIdx.x * 8; c < span.tail; c += CE_THREADS * 8) *reinterpret_cast<uint4*>(x + c) = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < edge; i += CE_THREADS) x[i < span.head ? i : span.tail + i - span.head] = __float2bfloat16(0.f);
    return;
  }
  const float scale = scale_ptr[0], l = lse[row];
  const long long local = label - vocab_start;
  const int mark = local >= 0 && local < cols ? int(local) : -1;
  auto grad = [&](float v, int c) {
    float p = expf(v - l);  // (not __expf, whose error grows with |v - l| and, next to a label's -1, decides whole digits)
    if (c == mark) p -= 1.f;
    return p * scale;
  };
  if constexpr (U > 0)
    for (int c = span.head + threadIdx.x * 8; c < span.tail; c += U * CE_THREADS * 8) {
    uint4 raw[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int ck = c + k * CE_THREADS * 8;
      if (ck < span.tail) raw[k] = *reinterpret_cast<const uint4*>(x + ck);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int ck = c + k * CE_THREADS * 8;
      if (ck < span.tail) {
        float v[8];
        ce_unpack(raw[k], v);
        uint4 o;
        uint32_t* ow = &o.x;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(grad(v[2 * j], ck + 2 * j), grad(v[2 * j + 1], ck + 2 * j + 1));
          ow[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        *reinterpret_cast<uint4*>(x + ck) = o;
      }
    }
  }
  for (int i = threadIdx.x; i < edge; i += CE_THREADS) {
    const int c = i < span.head ? i : span.tail + i - span.head;
    x[c] = __float2bfloat16(grad(__bfloat162float(x[c]), c));
  }
}

}  // namespace tpb

extern "C" int tpb_ce_stats(const void* logits, const int64_t* labels, float* stats, int rows, int cols, long long ld,
                            int vocab_start, int ignore_index, void* stream_) {
  if (!logits || !labels || !stats || rows <= 0 || cols <= 0) return TPB_ERR_ARG;
#define LAUNCH(U)                                                                                    \
  tpb::ce_stats_kernel<U><<<rows, tpb::CE_THREADS, 0, static_cast<cudaStream_t>(stream_)>>>(          \
      static_cast<const tpb::bf16*>(logits), labels, stats, cols, ld, vocab_start, ignore_index)
  CE_DISPATCH(cols, LAUNCH);
#undef LAUNCH
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

extern "C" int tpb_ce_grad(void* logits, const int64_t* labels, const float* lse, int rows, int cols, long long ld,
                           int vocab_start, int ignore_index, const float* scale_ptr, void* stream_) {
  if (!logits || !labels || !lse || !scale_ptr || rows <= 0 || cols <= 0) return TPB_ERR_ARG;
#define LAUNCH(U)                                                                                    \
  tpb::ce_grad_kernel<U><<<rows, tpb::CE_THREADS, 0, static_cast<cudaStream_t>(stream_)>>>(           \
      static_cast<tpb::bf16*>(logits), labels, lse, cols, ld, vocab_start, ignore_index, scale_ptr)
  CE_DISPATCH(cols, LAUNCH);
#undef LAUNCH
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

// CTAs of tpb_ce_loss = partials (float2 each) it needs.
extern "C" int tpb_ce_loss_parts(int rows) { return (rows + tpb::CE_THREADS - 1) / tpb::CE_THREADS; }

// stats: fp32 [world][rows][4] as tpb_ce_stats writes them, one slice per rank; lse: fp32 [rows]; loss, n_valid: one fp32 each (n_valid
// is at least 1).
extern "C" int tpb_ce_loss(const float* stats, const int64_t* labels, float* lse, float* partials, float* loss, float* n_valid, int world, int rows,
                           int ignore_index, void* stream_) {
  if (!stats || !labels || !lse || !partials || !loss || !n_valid || world <= 0 || rows <= 0) return TPB_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(stats) & 15) || (reinterpret_cast<uintptr_t>(partials) & 7)) return TPB_ERR_ALIGN;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  const int parts = tpb_ce_loss_parts(rows);
  float2* part = reinterpret_cast<float2*>(partials);
  tpb::ce_loss_kernel<<<parts, tpb::CE_THREADS, 0, s>>>(reinterpret_cast<const float4*>(stats), labels, lse, part, world, rows, ignore_index);
  tpb::ce_mean_kernel<<<1, tpb::CE_THREADS, 0, s>>>(part, parts, loss, n_valid);
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}
