// Many-token bf16 GEMM on CTA pairs: out[t, f] = act(sum_k x[t, k] w[f, k] + bias[f]) + residual[t, f].
//
// Two CTAs on neighbouring SMs (a cluster of two) work on ONE tile of 256 tokens x BN features with
// tcgen05.mma.cta_group::2: each CTA loads 128 token rows and BN / 2 feature rows into its own shared memory, the leader
// issues the MMAs for both, and each CTA finds its 128 rows x BN columns of the product in its own TMEM.
//
// What bounds it and why pairs: one k-block (64) of a 128 x 256 single-CTA tile takes the tensor core 512 clocks and
// brings 48 KB into shared memory - 96 bytes per clock and SM, more than the L2 delivers to all SMs at once.  A pair tile
// of 256 x 256 needs 32 KB per CTA for the same 512 clocks (64 bytes per clock).  Measured against the single-CTA kernel, same
// results to the bit: 8192 x 32000 x 4096 and its two gradients 1649 -> 1368 us each (1.57 PFLOP/s; cuBLAS in a short run 1.69, in seconds-long loops 1.41),
// the projections of a 7B layer at 4000 tokens 297 -> 265 us on average, the 4096 x 4096 ones at 8192 tokens 213 -> 177 us.
// In seconds-long loops the card is at its power limit and every access costs time: results leave in whole 32-byte sectors (8192 x
// 11008 x 4096 601 -> 571 us, its weight gradient 617 -> 600; 8192 x 4096 x 4096 222 -> 214; 8192 x 2048 x 2048 66 -> 62 us).
//
// One CTA (192 threads), persistent over the pair's tiles:
//   warp 0    : TMA producer of this CTA's operand rows; completion is counted on the LEADER's barrier (no multicast)
//   warp 1    : leader only: one thread issues the MMAs; the commits signal the barriers of both CTAs
//   warps 2-5 : epilogue of this CTA's 128 rows, two TMEM accumulators so that it runs under the next tile's MMAs
// Every mbarrier wait is bounded; on expiry the CTA records a status code and drains.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <atomic>

#include "attention_sm100.cuh"
#include "gemm_pair.cuh"
#include "launch.cuh"
#include "ptx_sm100.cuh"
#include "tpb_api.h"

namespace tpb {

constexpr int GP_BM = 256;       // tokens of a pair tile (128 per CTA = TMEM lanes)
constexpr int GP_BK = 64;        // one 128-byte swizzled row per operand row and stage
constexpr int GP_THREADS = 192;
constexpr int GP_MAX_STAGES = 8;
constexpr uint32_t GP_MN_BLOCK = 64 * GP_BK * 2;  // one [64 k][64 rows] block of an MN-major operand
// Tiles are walked in bands of 8 token tiles x all feature tiles: the ~74 tiles in flight then span 8 token tiles and
// about 9 feature tiles, the smallest operand footprint in L2 that the number of pairs allows.
constexpr int GP_BAND = 8;

struct GpParams {
  int m_extent, n_extent, k_blocks, m_tiles, n_tiles;
  int ld_out, act, a_mn, b_mn;
  float bias_scale;
  __nv_bfloat16* out;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  uint32_t* status;
  size_t out_elems;
};

// ---- CTA-pair forms of the tcgen05 / mbarrier / TMA instructions ----
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t mapa_u32(uint32_t addr, uint32_t rank) {  // `addr` in the shared memory of CTA `rank` of the cluster
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// Load into this CTA's shared memory, completion counted on a barrier of the pair's leader.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t leader_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on the barrier at this offset in BOTH CTAs once all MMAs issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"(uint16_t(3))
               : "memory");
}

__device__ __forceinline__ float gp_gelu_tanh(float x) {
  return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
}
__device__ __noinline__ float gp_act_call(float x, int act) {
  switch (act) {
    case 1: return fmaxf(x, 0.f);
    case 2: return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
    case 3: return gp_gelu_tanh(x);
    case 4: return x / (1.f + __expf(-x));
    default: return x;
  }
}

template <int BN>
struct GpShape {
  static constexpr int STAGES = BN == 256 ? 6 : 8;  // 192 KB: leaves room for a small collective kernel beside the GEMM
  static constexpr uint32_t A_BYTES = 128 * GP_BK * 2;
  static constexpr uint32_t B_BYTES = BN / 2 * GP_BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr size_t SMEM = size_t(STAGES) * STAGE_BYTES + 1024 /*align*/ + (2 * GP_MAX_STAGES + 4) * 8 + 16;
};

// (register cap of two CTAs per SM: see the many-token note in gemm_sm100.cu - a collective kernel may run beside this one)
template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 2)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const GpParams p) {
  using S = GpShape<BN>;
  constexpr uint32_t TMEM_COLS = 2 * BN;
  extern __shared__ uint8_t gp_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gp_smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + size_t(S::STAGES) * S::STAGE_BYTES);  // used in the leader
  uint64_t* empty_bar = full_bar + GP_MAX_STAGES;
  uint64_t* acc_full = empty_bar + GP_MAX_STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;              // [2], used in the leader
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();  // 0 = leader
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int tiles = p.m_tiles * p.n_tiles;

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], 8);  // one arrival per epilogue warp of either CTA
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  auto tile_at = [&](int t, int& mt, int& nt) {
    const int band = t / (GP_BAND * p.n_tiles), r = t - band * GP_BAND * p.n_tiles;
    const int rows = min(GP_BAND, p.m_tiles - band * GP_BAND);
    mt = band * GP_BAND + r % rows;
    nt = r / rows;
  };
  auto give_up = [&]() {
    atomicMax(p.status, STATUS_TIMEOUT_MBAR);
    *abort_flag = 1;
  };

  if (warp == 0) {
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; ok && t < tiles; t += pairs) {
        int mt, nt;
        tile_at(t, mt, nt);
        const int m0 = mt * GP_BM + int(rank) * 128, n0 = nt * BN + int(rank) * (BN / 2);
        for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
          const int s = it % S::STAGES;
          if (*abort_flag || !mbar_wait(&empty_bar[s], ((it / S::STAGES) & 1) ^ 1)) {
            give_up();
            ok = false;
            break;
          }
          uint8_t* a_dst = smem + size_t(s) * S::STAGE_BYTES;
          uint8_t* b_dst = a_dst + S::A_BYTES;
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
          if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * S::STAGE_BYTES);  // both CTAs' bytes
          if (p.a_mn) {
#pragma unroll
            for (int b = 0; b < 2; ++b) tma_load_2d_pair(a_dst + b * GP_MN_BLOCK, &tmap_a, bar, m0 + b * 64, kb * GP_BK);
          } else {
            tma_load_2d_pair(a_dst, &tmap_a, bar, kb * GP_BK, m0);
          }
          if (p.b_mn) {
#pragma unroll
            for (int b = 0; b < BN / 128; ++b) tma_load_2d_pair(b_dst + b * GP_MN_BLOCK, &tmap_b, bar, n0 + b * 64, kb * GP_BK);
          } else {
            tma_load_2d_pair(b_dst, &tmap_b, bar, kb * GP_BK, n0);
          }
        }
      }
      // the leader's last commits still arrive on this CTA's barriers: stay until each used stage has been released
      for (uint32_t i = it > uint32_t(S::STAGES) ? it - S::STAGES : 0; ok && i < it; ++i) {
        if (!mbar_wait(&empty_bar[i % S::STAGES], (i / S::STAGES) & 1)) {
          give_up();
          ok = false;
        }
      }
    }
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      const uint32_t idesc = make_idesc_bf16(GP_BM, BN, p.a_mn != 0, p.b_mn != 0);
      uint32_t it = 0, local = 0;
      bool ok = true;
      for (int t = pair; ok && t < tiles; t += pairs, ++local) {
        const int acc = local & 1;
        if (*abort_flag || !mbar_wait(&acc_empty[acc], ((local >> 1) & 1) ^ 1)) {
          give_up();
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < p.k_blocks; ++kb, ++it) {
          const int s = it % S::STAGES;
          if (!mbar_wait(&full_bar[s], (it / S::STAGES) & 1)) {
            give_up();
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + size_t(s) * S::STAGE_BYTES), b_addr = a_addr + S::A_BYTES;
#pragma unroll
          for (int kk = 0; kk < GP_BK / 16; ++kk) {
            // K-major: 16 elements are 32 bytes further along the rows; MN-major: 16 k-rows of 128 bytes further down
            const uint64_t adesc = p.a_mn ? make_desc_mnmajor_sw128(a_addr + kk * 16 * 128, GP_MN_BLOCK) : make_desc_kmajor_sw128(a_addr + kk * 32);
            const uint64_t bdesc = p.b_mn ? make_desc_mnmajor_sw128(b_addr + kk * 16 * 128, GP_MN_BLOCK) : make_desc_kmajor_sw128(b_addr + kk * 32);
            umma_bf16_pair(d_tmem, adesc, bdesc, idesc, (kb | kk) ? 1u : 0u);
          }
          umma_commit_pair(&empty_bar[s]);
        }
        if (ok) umma_commit_pair(&acc_full[acc]);
      }
    }
  } else {
    const int quarter = warp & 3;  // TMEM lane quarter this warp may access
    const int row = quarter * 32 + lane;
    const uint32_t acc_empty_leader[2] = {mapa_u32(smem_u32(&acc_empty[0]), 0), mapa_u32(smem_u32(&acc_empty[1]), 0)};
    const int out_cols = p.act == 5 ? 16 : 32;  // output columns of one 32-column chunk of the product
    const bool vec = (p.ld_out & 7) == 0 && !(reinterpret_cast<uintptr_t>(p.out) & 15) && !(reinterpret_cast<uintptr_t>(p.bias) & 15) &&
                     !(reinterpret_cast<uintptr_t>(p.residual) & 15);
    const bool sectors = vec && (p.ld_out & 15) == 0 && !(reinterpret_cast<uintptr_t>(p.out) & 31);
    uint32_t local = 0;
    for (int t = pair; t < tiles; t += pairs, ++local) {
      int mt, nt;
      tile_at(t, mt, nt);
      const int m = mt * GP_BM + int(rank) * 128 + row;
      const int acc = local & 1;
      const bool ready = !*abort_flag && mbar_wait(&acc_full[acc], (local >> 1) & 1);
      if (!__all_sync(0xffffffffu, ready)) {
        if (lane == 0) give_up();
        break;
      }
      tc_fence_after();
      const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16) + acc * BN;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        const int n0 = nt * BN + c0;
        if (n0 >= p.n_extent) break;
        uint32_t r[32];
        __syncwarp();  // (rows past the end skip the rest of a chunk)
        tmem_ld_x32(t_lane + c0, r);
        tmem_ld_wait();
        if (m >= p.m_extent) continue;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
        const size_t base = size_t(m) * p.ld_out + (p.act == 5 ? n0 >> 1 : n0);
        if (vec && n0 + 32 <= p.n_extent) {
          if (p.bias) {
            const uint4* bp = reinterpret_cast<const uint4*>(p.bias + n0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 b4 = __ldg(bp + q);
              const uint32_t bw[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                v[8 * q + 2 * j] += p.bias_scale * bf16_bits_to_float(bw[j] & 0xFFFF);
                v[8 * q + 2 * j + 1] += p.bias_scale * bf16_bits_to_float(bw[j] >> 16);
              }
            }
          }
          if (p.act == 5) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = v[j] / (1.f + __expf(-v[j])) * v[16 + j];
          } else if (p.act == 1) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
          } else if (p.act == 2) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0.5f * v[j] * (1.f + erff(v[j] * 0.70710678118654752f));
          } else if (p.act == 3) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = gp_gelu_tanh(v[j]);
          } else if (p.act == 4) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = v[j] / (1.f + __expf(-v[j]));
          }
          if (p.residual) {
            const uint4* rp = reinterpret_cast<const uint4*>(p.residual + base);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const uint4 r4 = rp[q];
              const uint32_t rw[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                v[8 * q + 2 * j] += bf16_bits_to_float(rw[j] & 0xFFFF);
                v[8 * q + 2 * j + 1] += bf16_bits_to_float(rw[j] >> 16);
              }
            }
          }
          if (TPB_IN_BOUNDS(base + out_cols <= p.out_elems, p.status)) {
            uint32_t w[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
            if (sectors) {
              st_global_v8(p.out + base, w);
              if (out_cols == 32) st_global_v8(p.out + base + 16, w + 8);
            } else {
              uint4* op = reinterpret_cast<uint4*>(p.out + base);
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                if (q * 8 < out_cols) op[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
              }
            }
          }
        } else if (p.act == 5) {  // (the feature count is a multiple of 32: only the vector path's alignment can be missing)
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float gte = v[j] + (p.bias ? p.bias_scale * __bfloat162float(p.bias[n0 + j]) : 0.f);
            const float upv = v[16 + j] + (p.bias ? p.bias_scale * __bfloat162float(p.bias[n0 + 16 + j]) : 0.f);
            if (TPB_IN_BOUNDS(base + j < p.out_elems, p.status)) p.out[base + j] = __float2bfloat16(gte / (1.f + __expf(-gte)) * upv);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (n0 + j < p.n_extent) {
              float x = v[j] + (p.bias ? p.bias_scale * __bfloat162float(p.bias[n0 + j]) : 0.f);
              if (p.act) x = gp_act_call(x, p.act);
              if (p.residual) x += __bfloat162float(p.residual[base + j]);
              if (TPB_IN_BOUNDS(base + j < p.out_elems, p.status)) p.out[base + j] = __float2bfloat16(x);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc_empty_leader[acc]);  // both accumulator halves may be overwritten after 8 of these
    }
  }

  // both CTAs stay until nobody can touch the other's barriers or TMEM any more
  __syncwarp();
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  if (warp == 1) tmem_dealloc_pair(tmem_base, TMEM_COLS);
}

// [rows, cols] bf16, cols contiguous, row pitch ld elements; box = [box_rows][64 cols], 128-byte swizzle.
static int gp_tmap(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
  EncodeTiledFn fn = fa_encode_fn();
  if (!fn) return TPB_ERR_DRIVER;
  cuuint64_t dims[2] = {cols, rows}, strides[1] = {ld * 2};
  cuuint32_t box[2] = {64, box_rows}, estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? TPB_OK
             : TPB_ERR_TMAP;
}

template <int BN>
static int gp_launch(const PairGemm& g, int sms, cudaStream_t stream) {
  using S = GpShape<BN>;
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TPB_ERR_CUDA;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(gemm_pair_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(S::SMEM)) != cudaSuccess) return TPB_ERR_CUDA;
    configured[dev].store(true, std::memory_order_release);
  }
  CUtensorMap ta, tb;
  int rc = g.x_mn ? gp_tmap(&ta, g.x, g.k, g.tokens, g.ldx, GP_BK) : gp_tmap(&ta, g.x, g.tokens, g.k, g.ldx, 128);
  if (rc == TPB_OK) rc = g.w_mn ? gp_tmap(&tb, g.w, g.k, g.features, g.ldw, GP_BK) : gp_tmap(&tb, g.w, g.features, g.k, g.ldw, BN / 2);
  if (rc != TPB_OK) return rc;
  GpParams p;
  memset(&p, 0, sizeof(p));
  p.m_extent = g.tokens;
  p.n_extent = g.features;
  p.k_blocks = (g.k + GP_BK - 1) / GP_BK;
  p.m_tiles = (g.tokens + GP_BM - 1) / GP_BM;
  p.n_tiles = (g.features + BN - 1) / BN;
  p.ld_out = g.ld_out;
  p.act = g.act;
  p.a_mn = g.x_mn;
  p.b_mn = g.w_mn;
  p.bias_scale = g.bias_scale;
  p.out = g.out;
  p.bias = g.bias;
  p.residual = g.residual;
  p.status = g.status;
  p.out_elems = g.out_elems;
  const long long tiles = (long long)p.m_tiles * p.n_tiles;
  const int pairs = int(tiles < sms / 2 ? tiles : sms / 2);
  return launch_kernel(gemm_pair_kernel<BN>, dim3(2 * pairs), dim3(GP_THREADS), S::SMEM, stream, ta, tb, p) == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

// Cost of a shape = rounds of tiles x time of one k-block of a tile, in clocks: the tensor core needs BN * 2 for a pair tile
// (BN = 256: 512), the operand bytes of a CTA arrive at about 70 per clock when all SMs load (pair 256: 468, pair 128: 351,
// single 256: 702, single 128: 468).  Against the fastest of the three over 66 to 4096 tokens and nine projections from 768 x 768 to
// 11008 x 4096, the choice is at most 9 % off, and more than 2 % off in 6 of 120 shapes; e.g. 128 x 4096 x 4096 single 26 us, pair 128 19 us,
// pair 256 25 us; 1024 x 4096 x 4096 49, 36, 27 us; 257 x 11008 x 4096 49, 51, 50 us.
int gemm_pair_tile(int tokens, int features, int sms) {
  auto rounds = [](long long tiles, int slots) { return (tiles + slots - 1) / slots; };
  auto tiles = [&](int bm, int bn) { return (long long)((tokens + bm - 1) / bm) * ((features + bn - 1) / bn); };
  const long long pair256 = rounds(tiles(256, 256), sms / 2) * 512, pair128 = rounds(tiles(256, 128), sms / 2) * 351;
  const bool wide = features >= 256 && tiles(128, 256) >= sms;  // what the single-CTA planner takes
  const long long single = wide ? rounds(tiles(128, 256), sms) * 702 : rounds(tiles(128, 128), sms) * 468;
  if (pair256 <= pair128 && pair256 <= single) return 256;
  if (pair128 <= single) return 128;
  return 0;
}

int gemm_pair_launch(const PairGemm& g, int bn, int sms, cudaStream_t stream) {
  return bn == 256 ? gp_launch<256>(g, sms, stream) : (bn == 128 ? gp_launch<128>(g, sms, stream) : int(TPB_ERR_ARG));
}

cudaError_t gemm_pair_preload() {
  cudaFuncAttributes attr;
  const cudaError_t e = cudaFuncGetAttributes(&attr, gemm_pair_kernel<256>);
  return e != cudaSuccess ? e : cudaFuncGetAttributes(&attr, gemm_pair_kernel<128>);
}

}  // namespace tpb
