// Few-token bf16 GEMM (decode): out[t, f] = act(norm(x)[t] . w[f] + bias[f]) + residual[t, f] for at most 64 tokens.
//
// Nothing but the stream of weights matters here: every weight byte is read from HBM once and used for a handful of tokens.
// What the time goes to besides those bytes, and what this kernel does about it:
//   * SMs without work, or with twice the work of the others.  128-row tiles leave 52 of 148 SMs idle at 12288 rows and make
//     24 SMs stream a second tile at 22016 rows; a 4096-row matrix needed split-K (park, fence, counter, re-read: 3 to 4 us)
//     to use more than 32 SMs.  Here the rows are dealt out in units of 32: every CTA owns one contiguous range, 1 to n units,
//     and no CTA ever needs another one's partial sums.
//   * Launch latency, barrier and TMEM set-up, and the first DRAM round trip, about 6 us per kernel in a chain.  With `early`
//     the kernel is launched as a programmatic dependent: it may start while its predecessor drains, and since the weights
//     do not depend on the predecessor, it fills its shared-memory ring with them BEFORE griddepcontrol.wait.  Only the
//     activations (x, residual, norm rows) and all stores come after the wait.
// A decode step of four 7B layers and the head (batch 8, 2048-token context) went from 793 to 691 us with this kernel and the
// early launches, a two-layer step of width 256 from 81 to 47 us.
//
// One CTA (192 threads): warp 0 = TMA producer, warp 1 = MMA issuer, warps 2-5 = epilogue.  The CTA walks its rows in passes
// of up to 128: weight rows fill the TMEM lanes (tcgen05.mma with M = 64 for passes of at most 64 rows - half the
// shared-memory reads per weight row - else 128), tokens are the N = 16 / 32 / 64 columns.  Rows of the MMA past the pass
// multiply whatever lies behind it in shared memory; their results are never read.
// Every mbarrier wait is bounded; on expiry the CTA records a status code and drains.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <atomic>

#include "attention_sm100.cuh"
#include "gemm_stream.cuh"
#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "tpb_api.h"

namespace tpb {

constexpr int GS_UNIT = 32;      // rows of a unit = rows of a weight box; the gated activation pairs 16 gate rows with their 16 up rows
constexpr int GS_BK = 64;        // columns of a box: 128-byte swizzled rows
constexpr int GS_KBOX = 4;       // boxes per stage and unit: 512 contiguous bytes of every weight row
constexpr int GS_THREADS = 192;
constexpr int GS_EPI = 128;
constexpr int GS_MAX_STAGES = 16;
constexpr int GS_PASS_UNITS = 4;

struct GsParams {
  int features, tokens, k_stages, units;
  int pass_units;       // units of the longest pass of any CTA: the shared-memory layout of a stage follows it
  int stages, early;
  int ld_out, act;
  float bias_scale;
  __nv_bfloat16* out;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  int norm_mode;
  float norm_eps;
  const __nv_bfloat16* norm_x;
  long long norm_ld;
  int norm_k;
  const float* norm_rowsum;
  uint32_t* status;
  size_t out_elems;
};

// (out of line: the epilogue runs once or twice per CTA, from a cold instruction cache - small code is fast code)
__device__ __noinline__ float gs_act(float x, int act) {
  switch (act) {
    case 1: return fmaxf(x, 0.f);
    case 2: return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
    case 3: return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
    case 4: return x / (1.f + __expf(-x));
    default: return x;
  }
}

// NACC accumulators per pass: consecutive MMAs into the same TMEM columns serialise, and one with N = 16 or 32 is far
// shorter than that latency, so k-steps are dealt round-robin and the epilogue adds the accumulators up.
template <int BN, int NACC>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const GsParams p) {
  constexpr uint32_t X_BOX = BN * GS_BK * 2, X_BYTES = GS_KBOX * X_BOX;
  constexpr uint32_t ACC_COLS = NACC * BN, TMEM_COLS = 2 * ACC_COLS;  // two accumulator sets: a pass's epilogue runs under the next
  static_assert(TMEM_COLS <= 512 && (TMEM_COLS & (TMEM_COLS - 1)) == 0 && TMEM_COLS >= 32, "TMEM allocation");
  const uint32_t w_box = uint32_t(p.pass_units) * GS_UNIT * 128;  // [rows of a pass][64 columns]
  const uint32_t w_bytes = GS_KBOX * w_box, stage_bytes = w_bytes + X_BYTES;

  extern __shared__ uint8_t gs_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gs_smem_raw) + 1023) & ~uintptr_t(1023));
  // control block first; the ring (and the rows that an MMA reads past its pass) behind it
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty_bar = full_bar + GS_MAX_STAGES;
  uint64_t* acc_full = empty_bar + GS_MAX_STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* norm_stats = reinterpret_cast<float*>(tmem_slot + 4);  // [64][rstd, mean * rstd]
  uint8_t* ring = smem + 1024;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit0 = int((long long)blockIdx.x * p.units / gridDim.x), unit1 = int((long long)(blockIdx.x + 1) * p.units / gridDim.x);
  const int passes = (unit1 - unit0 + GS_PASS_UNITS - 1) / GS_PASS_UNITS;
  auto pass_units = [&](int i) { return min(GS_PASS_UNITS, unit1 - unit0 - i * GS_PASS_UNITS); };

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_w);
    prefetch_tmap(&tmap_x);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], GS_EPI / 32);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (!p.early) pdl_wait();

  auto give_up = [&]() {
    atomicMax(p.status, STATUS_TIMEOUT_MBAR);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (elect_one()) {
      const int total = passes * p.k_stages;
      auto load_w = [&](int it) {
        const int pass = it / p.k_stages, ks = it - pass * p.k_stages, u = pass_units(pass);
        uint8_t* dst = ring + size_t(it % p.stages) * stage_bytes;
        uint64_t* bar = &full_bar[it % p.stages];
        mbar_expect_tx(bar, GS_KBOX * uint32_t(u) * GS_UNIT * 128 + X_BYTES);
        const int row0 = (unit0 + pass * GS_PASS_UNITS) * GS_UNIT;
        for (int i = 0; i < u; ++i) {
#pragma unroll
          for (int j = 0; j < GS_KBOX; ++j)  // (columns and rows past the end arrive as zeros)
            tma_load_2d(dst + j * w_box + i * GS_UNIT * 128, &tmap_w, bar, (ks * GS_KBOX + j) * GS_BK, row0 + i * GS_UNIT);
        }
      };
      auto load_x = [&](int it) {
        const int ks = it % p.k_stages;
        uint8_t* dst = ring + size_t(it % p.stages) * stage_bytes + w_bytes;
#pragma unroll
        for (int j = 0; j < GS_KBOX; ++j) tma_load_2d(dst + j * X_BOX, &tmap_x, &full_bar[it % p.stages], (ks * GS_KBOX + j) * GS_BK, 0);
      };
      const int ahead = min(total, p.stages);
      for (int it = 0; it < ahead; ++it) load_w(it);
      pdl_wait();
      pdl_trigger();
      for (int it = 0; it < ahead; ++it) load_x(it);
      for (int it = ahead; it < total; ++it) {
        if (*abort_flag || !mbar_wait(&empty_bar[it % p.stages], ((it / p.stages) & 1) ^ 1)) {
          give_up();
          break;
        }
        load_w(it);
        load_x(it);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      int it = 0;
      for (int pass = 0; pass < passes; ++pass) {
        const int acc = pass & 1;
        if (*abort_flag || !mbar_wait(&acc_empty[acc], ((pass >> 1) & 1) ^ 1)) {
          give_up();
          break;
        }
        tc_fence_after();
        const int u = pass_units(pass);
        const uint32_t idesc = make_idesc_bf16((u * GS_UNIT <= 64 && p.act != 5) ? 64 : 128, BN);
        const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
        uint32_t issued = 0;
        bool ok = true;
        for (int ks = 0; ks < p.k_stages; ++ks, ++it) {
          const int s = it % p.stages;
          if (!mbar_wait(&full_bar[s], (it / p.stages) & 1)) {
            give_up();
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t w_addr = smem_u32(ring + size_t(s) * stage_bytes), x_addr = w_addr + w_bytes;
#pragma unroll
          for (int j = 0; j < GS_KBOX; ++j) {
#pragma unroll
            for (int kk = 0; kk < GS_BK / 16; ++kk) {
              umma_bf16(d_tmem + (issued % NACC) * BN, make_desc_kmajor_sw128(w_addr + j * w_box + kk * 32),
                        make_desc_kmajor_sw128(x_addr + j * X_BOX + kk * 32), idesc, issued >= NACC ? 1u : 0u);
              ++issued;
            }
          }
          umma_commit(&empty_bar[s]);
        }
        if (!ok) break;
        umma_commit(&acc_full[acc]);
      }
    }
  } else {
    // ---------------- epilogue warps ----------------
    const int quarter = warp & 3;
    const bool gated = p.act == 5;
    pdl_wait();
    if (p.norm_mode) {
      // statistics of every token's unnormalised row, while the weights stream in
      const int chunks = p.norm_k >> 3;
      const float inv_k = 1.f / float(p.norm_k);
      for (int t = warp - 2; t < p.tokens; t += GS_EPI / 32) {
        const uint4* xrow = reinterpret_cast<const uint4*>(p.norm_x + size_t(t) * p.norm_ld);
        float s1 = 0.f, s2 = 0.f;
#pragma unroll 8
        for (int c = lane; c < chunks; c += 32) {
          const uint4 u = xrow[c];
          const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float lo = bf16_bits_to_float(w4[i] & 0xFFFF), hi = bf16_bits_to_float(w4[i] >> 16);
            s1 += lo + hi;
            s2 += lo * lo + hi * hi;
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          s1 += __shfl_xor_sync(0xffffffffu, s1, o);
          s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        if (lane == 0) {
          const float mean = p.norm_mode == 2 ? s1 * inv_k : 0.f;
          const float rstd = rsqrtf(fmaxf(s2 * inv_k - mean * mean, 0.f) + p.norm_eps);
          norm_stats[2 * t] = rstd;
          norm_stats[2 * t + 1] = mean * rstd;
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(GS_EPI) : "memory");
    }
    for (int pass = 0; pass < passes; ++pass) {
      const int acc = pass & 1, rows = pass_units(pass) * GS_UNIT;
      const bool m64 = rows <= 64 && !gated;
      // TMEM lane -> row of the pass: lane for M = 128; with M = 64 the first 16 lanes of each quarter hold 16 rows
      const int local_row = m64 ? quarter * 16 + lane : quarter * 32 + lane;
      const int m = (unit0 + pass * GS_PASS_UNITS) * GS_UNIT + local_row;
      const bool m_ok = local_row < rows && (!m64 || lane < 16) && m < p.features;
      // fetched while the weights are still streaming: a load behind the accumulators would add a full round trip
      const float bias = (p.bias && m_ok) ? p.bias_scale * __bfloat162float(p.bias[m]) : 0.f;
      const float rowsum = (p.norm_rowsum && m_ok) ? p.norm_rowsum[m] : 0.f;
      float res[16];
#pragma unroll
      for (int j = 0; j < 16; ++j)
        res[j] = (p.residual && m_ok && j < p.tokens) ? __bfloat162float(p.residual[size_t(j) * p.ld_out + m]) : 0.f;
      const bool ready = !*abort_flag && mbar_wait(&acc_full[acc], (pass >> 1) & 1);
      if (!__all_sync(0xffffffffu, ready)) {
        if (lane == 0) give_up();
        break;
      }
      tc_fence_after();
      const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16) + acc * ACC_COLS;
      const int n_acc = min(NACC, p.k_stages * GS_KBOX * (GS_BK / 16));
      const bool pitch_even = (p.ld_out & 1) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 3) == 0;
#pragma unroll 1
      for (int n0 = 0; n0 < BN; n0 += 16) {
        if (n0 >= p.tokens) break;
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
        __syncwarp();
#pragma unroll 1
        for (int a = 0; a < n_acc; ++a) {
          uint32_t r[16];
          tmem_ld_x16(t_lane + a * BN + n0, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] += __uint_as_float(r[j]);
        }
        if (n0 > 0 && p.residual) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            res[j] = (m_ok && n0 + j < p.tokens) ? __bfloat162float(p.residual[size_t(n0 + j) * p.ld_out + m]) : 0.f;
        }
        // a lane owns one feature: neighbouring lanes pair up so that every store carries two features (4 bytes)
        const bool writes_pair = pitch_even && !(lane & 1) && m + 1 < p.features;
        const bool covered = pitch_even && (lane & 1);  // the even neighbour stores this lane's value
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int t = n0 + j;
          if (t >= p.tokens) break;  // (uniform)
          float x = v[j];
          if (p.norm_mode) x = x * norm_stats[2 * t] - norm_stats[2 * t + 1] * rowsum;
          x += bias;
          if (gated) {
            // lanes 0-15 of a warp hold gate rows, lanes 16-31 the matching up rows
            const float partner = __shfl_xor_sync(0xffffffffu, x, 16);
            const size_t idx = size_t(t) * p.ld_out + (m >> 5) * 16 + (m & 15);
            if (m_ok && lane < 16 && TPB_IN_BOUNDS(idx < p.out_elems, p.status)) p.out[idx] = __float2bfloat16(x / (1.f + __expf(-x)) * partner);
            continue;
          }
          if (p.act) x = gs_act(x, p.act);
          x += res[j];
          const float up = __shfl_down_sync(0xffffffffu, x, 1);
          const size_t idx = size_t(t) * p.ld_out + m;
          if (m_ok && TPB_IN_BOUNDS(idx + (writes_pair ? 1 : 0) < p.out_elems, p.status)) {
            if (writes_pair) *reinterpret_cast<uint32_t*>(p.out + idx) = pack_bf16x2(x, up);
            else if (!covered) p.out[idx] = __float2bfloat16(x);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

static int g_stream_ring_kb = 160;
extern "C" int tpb_gemm_stream_tune(int ring_kb) {
  g_stream_ring_kb = ring_kb;
  return TPB_OK;
}

static int gs_tmap(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
  EncodeTiledFn fn = fa_encode_fn();
  if (!fn) return TPB_ERR_DRIVER;
  cuuint64_t dims[2] = {cols, rows}, strides[1] = {ld * 2};
  cuuint32_t box[2] = {GS_BK, box_rows}, estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? TPB_OK
             : TPB_ERR_TMAP;
}

template <int BN, int NACC>
static int gs_launch(const StreamGemm& g, int sms, cudaStream_t stream) {
  GsParams p;
  memset(&p, 0, sizeof(p));
  p.features = g.features;
  p.tokens = g.tokens;
  p.k_stages = (g.k + GS_KBOX * GS_BK - 1) / (GS_KBOX * GS_BK);
  p.units = (g.features + GS_UNIT - 1) / GS_UNIT;
  const int grid = p.units < sms ? p.units : sms;
  const int most = (p.units + grid - 1) / grid;  // units of the CTA with the longest range
  p.pass_units = most < GS_PASS_UNITS ? most : GS_PASS_UNITS;
  const size_t stage_bytes = size_t(GS_KBOX) * (size_t(p.pass_units) * GS_UNIT * 128 + BN * GS_BK * 2);
  // an MMA of M = 64 / 128 rows reads that many rows from the last box of the ring: up to 12 KB behind it
  const size_t over = size_t(GS_UNIT) * 128 * (GS_PASS_UNITS - 1);
  int stages = int((size_t(g_stream_ring_kb) * 1024) / stage_bytes);
  if (stages > GS_MAX_STAGES) stages = GS_MAX_STAGES;
  if (stages < 2) stages = 2;
  p.stages = stages;
  const size_t smem = 1024 + 1024 + stages * stage_bytes + over;
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TPB_ERR_CUDA;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(gemm_stream_kernel<BN, NACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return TPB_ERR_CUDA;
    configured[dev].store(true, std::memory_order_release);
  }
  CUtensorMap tw, tx;
  int rc = gs_tmap(&tw, g.w, g.features, g.k, g.ldw, GS_UNIT);
  if (rc == TPB_OK) rc = gs_tmap(&tx, g.x, g.tokens, g.k, g.ldx, BN);
  if (rc != TPB_OK) return rc;
  p.early = g.early;
  p.ld_out = g.ld_out;
  p.act = g.act;
  p.bias_scale = g.bias_scale;
  p.out = g.out;
  p.bias = g.bias;
  p.residual = g.residual;
  p.norm_mode = g.norm_mode;
  p.norm_eps = g.norm_eps;
  p.norm_x = g.norm_x;
  p.norm_ld = g.norm_ld;
  p.norm_k = g.norm_k;
  p.norm_rowsum = g.norm_rowsum;
  p.status = g.status;
  p.out_elems = g.out_elems;
  return launch_dependent(gemm_stream_kernel<BN, NACC>, dim3(grid), dim3(GS_THREADS), smem, stream, g.early != 0 || pdl_enabled(), tw, tx, p) == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

bool gemm_stream_fits(int features, int k, int sms) {
  const long long unit_bytes = 2LL * GS_UNIT * k;
  return (features + GS_UNIT - 1) / GS_UNIT >= sms / 2 || unit_bytes <= 1024 * 1024;
}

int gemm_stream_launch(const StreamGemm& g, int sms, cudaStream_t stream) {
  if (g.tokens <= 16) return gs_launch<16, 8>(g, sms, stream);
  if (g.tokens <= 32) return gs_launch<32, 8>(g, sms, stream);
  if (g.tokens <= 64) return gs_launch<64, 2>(g, sms, stream);
  return TPB_ERR_ARG;
}

cudaError_t gemm_stream_preload() {
  cudaFuncAttributes attr;
  cudaError_t e = cudaFuncGetAttributes(&attr, gemm_stream_kernel<16, 8>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, gemm_stream_kernel<32, 8>);
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, gemm_stream_kernel<64, 2>);
  return e;
}

}  // namespace tpb
