// Attention backward for sm_100a on tcgen05 tensor cores, with an optional additive score bias (scores = S * scale + bias;
// d(bias) = P * (dP - delta), summed over whatever dimensions the bias broadcasts over, comes from attn_bias_grad_kernel for a dense bf16
// bias that the batches share, and is otherwise added into an fp32 buffer by the dQ launch, which visits every (query, key) pair exactly once).
//
//   P  = exp(S * scale - lse)          S  = Q K^T
//   dV = P^T dO                        dP = dO V^T
//   dS = P * (dP - delta) * scale      delta[i] = sum_d out[i, d] * dout[i, d]
//   dQ = dS K                          dK = dS^T Q
//
// Two launches, dK / dV and dQ, and where it is taken that of the bias gradient, free of atomics and therefore deterministic (a bias gradient
// that the dQ launch adds up is the exception: fp32 atomic adds).  A CTA keeps 128 "resident" rows (the TMEM lanes) and streams the other sequence through.  There are two kernels, each a
// template of both launches: attn_bwd_tcgen05_kernel streams 64 rows per step (described here), attn_bwd_wide_kernel 128, or 64
// with two CTAs per SM (described there); two_per_sm and step_rows below say which launch takes which.
//
//   dK / dV (DKV = true) : resident = 128 keys of one KV head (K and V tiles), streamed = queries (Q and dO, over all
//                          query heads of the group):  S^T = K Q^T and dP^T = V dO^T land in TMEM with a key per lane,
//                          the elementwise warps turn them into P^T and dS^T (bf16, written back over their own
//                          columns), and dV += P^T dO, dK += dS^T Q read them from TENSOR MEMORY as the A operand, the
//                          streamed tile being the MN-major B operand as it lies in memory.
//   dQ (DKV = false)     : resident = 128 queries of one head (Q and dO), streamed = keys (K and V): S = Q K^T,
//                          dP = dO V^T, dQ += dS K.
//
//   warp 0    : TMA producer (resident tiles once, streamed tiles into a 3-deep ring; for dK / dV also the streamed
//               queries' log-sum-exp and delta into shared memory)
//   warp 1    : MMA issuer; the two score products of step n + 1 are issued BEFORE the wait for the elementwise warps
//               of step n (two TMEM buffers), so the tensor core always has work
//   warps 2-9 : elementwise - two threads per TMEM lane, one per half of the step's 64 columns
//
// TMEM (512 columns): S 2 x 64 | dP 2 x 64 | accumulator 0 (dK or dQ) | accumulator 1 (dV) | resident tiles (RES_TMEM).  Shared memory at head_dim
// 128: 2 x 32 KB resident + 3 x 2 x 16 KB streamed = 160 KB.  Every mbarrier wait is bounded; on expiry the CTA records
// a status code and drains.  No TMA load has a multicast qualifier.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <type_traits>

#include "attention_sm100.cuh"
#include "ptx_sm100.cuh"
#include "tpb_api.h"

namespace tpb {

typedef __nv_bfloat16 bf16;

constexpr int BW_R = 128;      // resident rows = TMEM lanes
constexpr int BW_T = 64;       // streamed rows per step = TMEM columns of one score buffer
constexpr int BW_STAGES = 3;
constexpr int BW_THREADS = 320;
constexpr int BW_BIAS_BYTES = BW_R * BW_T * 2;  // bias elements of one step
constexpr int BW_T_BLOCK_BYTES = BW_T * 128;  // one [64 rows][64 elements] swizzled block

struct BwParams {
  int sq, sk, q_heads, kv_heads, causal;
  float scale, scale_log2e;
  const float* lse;    // [batch][q_heads][sq], natural log
  const float* delta;  // [batch][q_heads][sq]
  bf16* out0;          // dK (DKV) or dQ
  long long o0_sb, o0_ss, o0_sh;
  bf16* out1;          // dV (DKV)
  long long o1_sb, o1_ss, o1_sh;
  const void* bias;    // additive score bias in natural-log units over (batch, head, query, key), element strides, 0 broadcasts
  int bias_kind;       // 0 none, 1 fp32, 2 bf16
  long long b_sb, b_sh, b_sq, b_sk;
  float* dbias;        // fp32, the bias' own strides, zero-initialised by the caller; written by the dQ launch only (or null)
  int bias_vec;        // bias rows readable as aligned vectors of eight keys (bias_vector_rows); so is dbias then
  float inv_scale;
  uint32_t* status;
};

// ---- what the elementwise warps of both kernels do with 32 columns (streamed rows) of one TMEM lane (resident row) ----

// Bits lo to hi - 1 of 32.
__device__ __forceinline__ uint32_t bw_bits(int lo, int hi) {
  uint32_t bits = 0xffffffffu;
  if (lo > 0) bits = lo < 32 ? bits << lo : 0u;
  if (hi < 32) bits = hi > 0 ? bits & (0xffffffffu >> (32 - hi)) : 0u;
  return bits;
}

// Bits of the columns from col0 on that are visible pairs with resident row ri; only steps that touch the diagonal or an end have any cleared.
template <bool DKV>
__device__ __forceinline__ uint32_t bw_visible(const BwParams& p, int ri, int shift, int col0) {
  int lo = 0, hi = 32;  // columns [lo, hi) are
  if (DKV) {
    if (ri >= p.sk) hi = 0;
    if (p.causal) lo = max(0, ri - shift - col0);  // query >= key - shift
  } else {
    hi = min(32, min(p.sk, p.causal ? ri + shift + 1 : p.sk) - col0);  // key <= query + shift
  }
  return bw_bits(lo, hi);
}

// Eight score biases of resident row `row` from column `col` of a step on, out of the step's tile in shared memory.
template <bool DKV>
__device__ __forceinline__ void bw_bias8(const uint8_t* tile, int row, int col, float (&v)[8]) {
  if (DKV) {  // column = query row of the tile, lanes read consecutive keys
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __bfloat162float(*reinterpret_cast<const bf16*>(tile + (col + i) * (BW_R * 2) + row * 2));
  } else {  // eight keys of this thread's query: one swizzled 16-byte chunk of a block of 64 keys
    const uint4 u = *reinterpret_cast<const uint4*>(tile + (col >> 6) * FA_BLOCK_BYTES + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4));
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
  }
}

// Adds the bias gradients of keys col to col + 3 of one query.
__device__ __forceinline__ void bw_add_dbias(const BwParams& p, long long bias_base, int col, const float (&db)[4]) {
  float* dst = p.dbias + bias_base + (long long)col * p.b_sk;
  if (p.bias_vec && col + 4 <= p.sk) {
    // the batches (and whatever else the bias broadcasts over) add into one buffer: four keys per reduction
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(db[0]), "f"(db[1]), "f"(db[2]), "f"(db[3]) : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (db[i] != 0.f && col + i < p.sk) atomicAdd(dst + i * p.b_sk, db[i]);
  }
}

// N accumulator columns as bf16: whole 32-byte sectors, 16 bytes or pairs, as the address allows.
template <int N>
__device__ __forceinline__ void bw_store_row(bf16* dst, const uint32_t (&o)[N]) {
  uint32_t w[N / 2];
#pragma unroll
  for (int i = 0; i < N / 2; ++i) w[i] = pack_bf16x2(__uint_as_float(o[2 * i]), __uint_as_float(o[2 * i + 1]));
  if ((reinterpret_cast<uintptr_t>(dst) & 31) == 0) {
#pragma unroll
    for (int i = 0; i < N / 2; i += 8) st_global_v8(dst + 2 * i, w + i);
  } else if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
    for (int i = 0; i < N / 2; i += 4) *reinterpret_cast<uint4*>(dst + 2 * i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < N / 2; ++i) *reinterpret_cast<uint32_t*>(dst + 2 * i) = w[i];
  }
}

// BIAS: the score-bias code exists only in the instantiations that need it.  1: elements are loaded by the threads that use them;
// 2: a dense bf16 bias whose rows TMA can address travels with the streamed tiles, [64 queries][128 keys] (dK / dV) or
// [128 queries][64 keys] (dQ) per step, so that no elementwise warp ever waits for a global load (16 x 512 tokens, 32 heads of 64,
// one bias for all batches, in steps of 64 rows: dK / dV 1093 -> 205 us, dQ 316 -> 231 us).
template <int D, bool DKV, int BIAS>
__global__ void __launch_bounds__(BW_THREADS, 1)
attn_bwd_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_r1, const __grid_constant__ CUtensorMap tmap_r2,
                        const __grid_constant__ CUtensorMap tmap_t1, const __grid_constant__ CUtensorMap tmap_t2,
                        const __grid_constant__ CUtensorMap tmap_b, const BwParams p) {
  constexpr int DB = D / 64;
  constexpr uint32_t R_BYTES = DB * FA_BLOCK_BYTES;    // one resident tile (128 rows)
  constexpr uint32_t T_BYTES = DB * BW_T_BLOCK_BYTES;  // one streamed tile (64 rows)
  constexpr uint32_t TMEM_COLS = 512;
  constexpr uint32_t S_COL0 = 0, DP_COL0 = 2 * BW_T, ACC0_COL = 4 * BW_T, ACC1_COL = 4 * BW_T + D;
  // The resident tiles as tensor-memory A operands where 512 columns leave room for them (all of dQ, dK / dV at head_dim 64): from
  // shared memory, a score MMA of 128 x 64 x 16 reads 6 KB for 32 clocks of work and is bound by that (in this kernel, dQ of 4 x 2048, 32
  // heads of 128, causal: 248 -> 233 us; whole backward of 16 x 512, 32 heads of 64: 291 -> 273 us).
  constexpr bool RES_TMEM = !DKV || D == 64;
  constexpr uint32_t RES_COL0 = ACC0_COL + (DKV ? 2 : 1) * D;  // resident 1, then resident 2: D / 2 columns each (two bf16 per column)
  static_assert(!RES_TMEM || RES_COL0 + D <= TMEM_COLS, "tensor memory columns");
  constexpr uint32_t IDESC_S = make_idesc_bf16(BW_R, BW_T, false, false);
  constexpr uint32_t IDESC_ACC = make_idesc_bf16(BW_R, D, false, true);

  extern __shared__ uint8_t bw_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(bw_smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* r1_s = smem;
  uint8_t* r2_s = r1_s + R_BYTES;
  uint8_t* t1_s = r2_s + R_BYTES;              // [stages]
  uint8_t* t2_s = t1_s + BW_STAGES * T_BYTES;  // [stages]
  // [stages][32 pairs of streamed queries]: {-lse * log2(e) of both (-inf = no such query), -delta * scale of both}
  float4* stat_s = reinterpret_cast<float4*>(t2_s + BW_STAGES * T_BYTES);
  uint8_t* bias_s = reinterpret_cast<uint8_t*>(t2_s + BW_STAGES * T_BYTES);  // [stages], BIAS == 2 only (1024-byte aligned for the swizzle)
  if (BIAS == 2) stat_s = reinterpret_cast<float4*>(bias_s + BW_STAGES * BW_BIAS_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(stat_s + BW_STAGES * BW_T / 2);
  uint64_t* r_full = bars;
  uint64_t* t_full = bars + 1;                   // [stages]
  uint64_t* t_empty = bars + 1 + BW_STAGES;      // [stages]
  uint64_t* s_full = bars + 1 + 2 * BW_STAGES;   // [2]
  uint64_t* p_full = s_full + 2;                 // [2]
  uint64_t* acc_full = p_full + 2;
  uint64_t* res_full = acc_full + 1;             // RES_TMEM: the resident tiles are in tensor memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (known to be uniform)
  const int b = blockIdx.z;
  const int shift = p.sk - p.sq;  // query i may see keys j <= i + shift when causal
  const int group = p.q_heads / p.kv_heads;
  // ---- what this CTA owns and which steps it walks (the same arithmetic in every role) ----
  int r0, head, kvh, step0, per_head, n_steps;
  if (DKV) {
    r0 = blockIdx.x * BW_R;  // first key; low key tiles see the most queries when causal, so they start first
    kvh = blockIdx.y;
    head = kvh * group;      // first query head of the group
    const int q_steps = (p.sq + BW_T - 1) / BW_T;
    step0 = p.causal ? max(0, r0 - shift) / BW_T : 0;  // first 64-query step with a query that sees key r0
    per_head = max(0, q_steps - step0);
    n_steps = per_head * group;
  } else {
    r0 = (gridDim.x - 1 - blockIdx.x) * BW_R;  // first query; late query tiles see the most keys when causal
    head = blockIdx.y;
    kvh = head / group;
    int kv_end = p.sk;
    if (p.causal) kv_end = min(p.sk, r0 + BW_R + shift);
    step0 = 0;
    per_head = kv_end > 0 ? (kv_end + BW_T - 1) / BW_T : 0;
    n_steps = per_head;
  }

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_r1);
    prefetch_tmap(&tmap_r2);
    prefetch_tmap(&tmap_t1);
    prefetch_tmap(&tmap_t2);
    mbar_init(r_full, 1);
    for (int s = 0; s < BW_STAGES; ++s) {
      mbar_init(&t_full[s], DKV ? 2 : 1);  // the TMA bytes, and for dK / dV the step's lse / delta written by the producer warp
      mbar_init(&t_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 8);  // one arrival per elementwise warp
    }
    mbar_init(acc_full, 1);
    mbar_init(res_full, 8);
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

  auto give_up = [&](uint32_t code) {
    atomicMax(p.status, code);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer (the whole warp stays together: all lanes write lse / delta) ----------------
    if (n_steps > 0) {
      if (lane == 0) {
        mbar_expect_tx(r_full, 2 * R_BYTES);
#pragma unroll
        for (int d = 0; d < DB; ++d) {
          tma_load_4d(r1_s + d * FA_BLOCK_BYTES, &tmap_r1, r_full, d * 64, r0, DKV ? kvh : head, b);
          tma_load_4d(r2_s + d * FA_BLOCK_BYTES, &tmap_r2, r_full, d * 64, r0, DKV ? kvh : head, b);
        }
      }
      int g = 0, local = 0;  // query head of the group (dK / dV), step within it
      for (int n = 0; n < n_steps; ++n) {
        const int s = n % BW_STAGES;
        const uint32_t par = ((n / BW_STAGES) & 1) ^ 1;
        const bool ok = !*abort_flag && mbar_wait(&t_empty[s], par);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0 && !*abort_flag) give_up(STATUS_TIMEOUT_MBAR);
          break;
        }
        const int row0 = (step0 + local) * BW_T;  // first streamed row of the step
        const int t_head = DKV ? head + g : kvh;
        if (++local == per_head) { local = 0; ++g; }
        if (lane == 0) {
          mbar_expect_tx(&t_full[s], 2 * T_BYTES + (BIAS == 2 ? BW_BIAS_BYTES : 0));
          if (BIAS == 2)
            tma_load_4d(bias_s + s * BW_BIAS_BYTES, &tmap_b, &t_full[s], DKV ? r0 : row0, DKV ? row0 : r0, p.b_sh ? (DKV ? t_head : head) : 0, p.b_sb ? b : 0);
#pragma unroll
          for (int d = 0; d < DB; ++d) {
            tma_load_4d(t1_s + s * T_BYTES + d * BW_T_BLOCK_BYTES, &tmap_t1, &t_full[s], d * 64, row0, t_head, b);
            tma_load_4d(t2_s + s * T_BYTES + d * BW_T_BLOCK_BYTES, &tmap_t2, &t_full[s], d * 64, row0, t_head, b);
          }
        }
        if (DKV) {
#pragma unroll
          for (int c = lane; c < BW_T; c += 32) {
            const int qi = row0 + c;
            float l2 = -INFINITY, dl = 0.f;
            if (qi < p.sq) {
              const long long idx = ((long long)b * p.q_heads + t_head) * p.sq + qi;
              const float l = __ldg(p.lse + idx);
              if (l != -INFINITY) l2 = -l * 1.4426950408889634f;  // (a query without a visible key has P = 0 everywhere)
              dl = -__ldg(p.delta + idx) * p.scale;
            }
            float* pair = reinterpret_cast<float*>(stat_s + s * (BW_T / 2) + (c >> 1)) + (c & 1);
            pair[0] = l2;
            pair[2] = dl;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&t_full[s]);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the warp stays together, one lane issues: see umma_bf16_lead) ----------------
    if (n_steps > 0) {
      const uint32_t leader = elect_one();
      const uint32_t r1_lo = desc_kmajor_lo(smem_u32(r1_s)), r2_lo = desc_kmajor_lo(smem_u32(r2_s));
      auto issue_scores = [&](int n) {  // S[n & 1] = R1 T1(n)^T, dP[n & 1] = R2 T2(n)^T
        const int s = n % BW_STAGES, buf = n & 1;
        const uint32_t t1_lo = desc_kmajor_lo(smem_u32(t1_s + s * T_BYTES)), t2_lo = desc_kmajor_lo(smem_u32(t2_s + s * T_BYTES));
#pragma unroll
        for (int d = 0; d < DB; ++d) {
#pragma unroll
          for (int kk = 0; kk < 64 / 16; ++kk)
            if (RES_TMEM)
              umma_bf16_tmem_a_lead(leader, tmem_base + S_COL0 + buf * BW_T, tmem_base + RES_COL0 + (d * 4 + kk) * 8,
                                    t1_lo + d * (BW_T_BLOCK_BYTES >> 4) + kk * 2, IDESC_S, (d | kk) ? 1u : 0u);
            else
              umma_bf16_lead(leader, tmem_base + S_COL0 + buf * BW_T, r1_lo + d * (FA_BLOCK_BYTES >> 4) + kk * 2,
                             t1_lo + d * (BW_T_BLOCK_BYTES >> 4) + kk * 2, IDESC_S, (d | kk) ? 1u : 0u);
        }
#pragma unroll
        for (int d = 0; d < DB; ++d) {
#pragma unroll
          for (int kk = 0; kk < 64 / 16; ++kk)
            if (RES_TMEM)
              umma_bf16_tmem_a_lead(leader, tmem_base + DP_COL0 + buf * BW_T, tmem_base + RES_COL0 + D / 2 + (d * 4 + kk) * 8,
                                    t2_lo + d * (BW_T_BLOCK_BYTES >> 4) + kk * 2, IDESC_S, (d | kk) ? 1u : 0u);
            else
              umma_bf16_lead(leader, tmem_base + DP_COL0 + buf * BW_T, r2_lo + d * (FA_BLOCK_BYTES >> 4) + kk * 2,
                             t2_lo + d * (BW_T_BLOCK_BYTES >> 4) + kk * 2, IDESC_S, (d | kk) ? 1u : 0u);
        }
        umma_commit_lead(leader, &s_full[buf]);
      };
      auto issue_accumulate = [&](int n) {
        const int s = n % BW_STAGES, buf = n & 1;
        const uint32_t t1_lo = desc_mnmajor_lo(smem_u32(t1_s + s * T_BYTES), BW_T_BLOCK_BYTES);
        const uint32_t t2_lo = desc_mnmajor_lo(smem_u32(t2_s + s * T_BYTES), BW_T_BLOCK_BYTES);
#pragma unroll
        for (int kk = 0; kk < BW_T / 16; ++kk) {
          // the bf16 operand of the 16 streamed rows kk: written by the thread that owns their column half, inside that half
          const uint32_t a_col = (kk >> 1) * 32 + (kk & 1) * 8;
          if (DKV)  // dV += P^T dO
            umma_bf16_tmem_a_lead(leader, tmem_base + ACC1_COL, tmem_base + S_COL0 + buf * BW_T + a_col, t2_lo + kk * (16 * 128 >> 4), IDESC_ACC,
                                  (n | kk) ? 1u : 0u);
          // dK += dS^T Q   or   dQ += dS K
          umma_bf16_tmem_a_lead(leader, tmem_base + ACC0_COL, tmem_base + DP_COL0 + buf * BW_T + a_col, t1_lo + kk * (16 * 128 >> 4), IDESC_ACC,
                                (n | kk) ? 1u : 0u);
        }
      };
      auto wait_all = [&](uint64_t* bar, uint32_t parity) {
        const bool there = __all_sync(0xffffffffu, mbar_wait(bar, parity));
        if (!there && leader) give_up(STATUS_TIMEOUT_MBAR);
        tc_fence_after();
        return there;
      };
      bool ok = wait_all(RES_TMEM ? res_full : r_full, 0) && wait_all(&t_full[0], 0);
      if (ok) issue_scores(0);
      for (int n = 0; ok && n < n_steps; ++n) {
        if (n + 1 < n_steps) {
          // scores of the next step: their TMEM buffer was last read by the accumulate MMAs of step n - 1 (issued
          // before these) and by the elementwise warps of step n - 1 (who delivered before those were issued)
          ok = wait_all(&t_full[(n + 1) % BW_STAGES], ((n + 1) / BW_STAGES) & 1);
          if (!ok) break;
          issue_scores(n + 1);
        }
        ok = wait_all(&p_full[n & 1], (n >> 1) & 1);
        if (!ok) break;
        issue_accumulate(n);
        umma_commit_lead(leader, &t_empty[n % BW_STAGES]);  // the streamed tiles of step n may be overwritten once these MMAs retire
      }
      umma_commit_lead(leader, acc_full);
    }
  } else {
    // ---------------- elementwise warps ----------------
    constexpr int HC = BW_T / 2;   // columns per thread and step
    constexpr int HD = D / 2;      // accumulator columns per thread in the epilogue
    const int quarter = warp & 3;  // TMEM lane quarter this warp may access
    const int half = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const int ri = r0 + row;  // key (DKV) or query
    const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16);
    float my_lse2 = -INFINITY, my_del = 0.f;  // negated
    if (!DKV && ri < p.sq) {
      const long long idx = ((long long)b * p.q_heads + head) * p.sq + ri;
      const float l = __ldg(p.lse + idx);
      if (l != -INFINITY) my_lse2 = -l * 1.4426950408889634f;
      my_del = -__ldg(p.delta + idx) * p.scale;
    }
    bool alive = true;
    int g = 0, local = 0;  // as in the producer
    if (RES_TMEM && n_steps > 0) {
      // resident tiles: swizzled shared memory -> tensor memory, a row per thread, one tile per half
      if (!mbar_wait(r_full, 0)) {
        give_up(STATUS_TIMEOUT_MBAR);
        alive = false;
      }
      const uint8_t* tile = half ? r2_s : r1_s;
#pragma unroll
      for (int d = 0; d < DB; ++d) {
        uint32_t w[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 u = *reinterpret_cast<const uint4*>(tile + d * FA_BLOCK_BYTES + row * 128 + ((c ^ (row & 7)) << 4));
          w[4 * c] = u.x; w[4 * c + 1] = u.y; w[4 * c + 2] = u.z; w[4 * c + 3] = u.w;
        }
        __syncwarp();
        tmem_st_x32(t_lane + RES_COL0 + half * (D / 2) + d * 32, w);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(res_full);
    }

    for (int n = 0; alive && n < n_steps; ++n) {
      const int s = n % BW_STAGES, buf = n & 1;
      if (*abort_flag || ((DKV || BIAS == 2) && !mbar_wait(&t_full[s], (n / BW_STAGES) & 1)) || !mbar_wait(&s_full[buf], (n >> 1) & 1)) {
        if (!*abort_flag) give_up(STATUS_TIMEOUT_MBAR);
        alive = false;
        break;
      }
      tc_fence_after();
      const int col0 = (step0 + local) * BW_T + half * HC;  // first query (DKV) or key of my columns
      const int b_head = DKV ? head + g : head;
      if (++local == per_head) { local = 0; ++g; }
      uint32_t sv[HC], dv[HC];
      tmem_ld_x32(t_lane + S_COL0 + buf * BW_T + half * HC, sv);
      tmem_ld_x32(t_lane + DP_COL0 + buf * BW_T + half * HC, dv);
      tmem_ld_wait();
      const uint32_t visible = bw_visible<DKV>(p, ri, shift, col0);
      const bool masked = __any_sync(0xffffffffu, visible != 0xffffffffu);  // (per warp: the common loop has no masks)
      // score bias: element (query, key) = (col0 + c, ri) for dK / dV - there the lanes of a warp own consecutive keys - and
      // (ri, col0 + c) for dQ, where a thread's columns are consecutive keys of one row and are read eight at a time
      const long long bias_base = BIAS ? (long long)b * p.b_sb + (long long)b_head * p.b_sh + (long long)ri * (DKV ? p.b_sk : p.b_sq) : 0;
      const long long bias_step = DKV ? p.b_sq : p.b_sk;  // per column
      const int col_limit = DKV ? p.sq : p.sk, row_limit = DKV ? p.sk : p.sq;
      uint32_t pp[HC / 2], ds[HC / 2];
      float bv[8], db[4];
      auto pairs = [&](auto with_masks) {
        constexpr bool MASKED = decltype(with_masks)::value;
#pragma unroll
        for (int c = 0; c < HC; c += 2) {
          float l0, l1, d0, d1;
          if (DKV) {
            const float4 st = stat_s[s * (BW_T / 2) + ((half * HC + c) >> 1)];
            l0 = st.x; l1 = st.y; d0 = st.z; d1 = st.w;
          } else {
            l0 = l1 = my_lse2;
            d0 = d1 = my_del;
          }
          if (BIAS == 2 && (c & 7) == 0) bw_bias8<DKV>(bias_s + s * BW_BIAS_BYTES, row, half * HC + c, bv);
          if (BIAS == 1 && (c & 7) == 0)
            load_bias8(p.bias, p.bias_kind, bias_base + (long long)(col0 + c) * bias_step, bias_step, ri < row_limit ? col_limit - col0 - c : 0,
                       !DKV && p.bias_vec, bv);
          float x0, x1, p0, p1, g0, g1;
          ffma2(x0, x1, __uint_as_float(sv[c]), __uint_as_float(sv[c + 1]), p.scale_log2e, p.scale_log2e, l0, l1);
          if (BIAS) {
            x0 += bv[c & 7] * 1.4426950408889634f;
            x1 += bv[(c & 7) + 1] * 1.4426950408889634f;
          }
          p0 = ex2_approx(x0);
          p1 = ex2_approx(x1);
          if (MASKED) {
            if (!(visible >> c & 1)) p0 = 0.f;
            if (!(visible >> (c + 1) & 1)) p1 = 0.f;
          }
          ffma2(g0, g1, __uint_as_float(dv[c]), __uint_as_float(dv[c + 1]), p.scale, p.scale, d0, d1);  // (dP - delta) * scale
          ffma2(g0, g1, g0, g1, p0, p1, 0.f, 0.f);
          if (BIAS && !DKV && p.dbias) {  // d(bias) = P (dP - delta) = dS / scale; pairs that are masked or out of range contribute nothing
            db[c & 3] = p0 != 0.f ? g0 * p.inv_scale : 0.f;
            db[(c & 3) + 1] = p1 != 0.f ? g1 * p.inv_scale : 0.f;
            if ((c & 3) == 2 && ri < row_limit) bw_add_dbias(p, bias_base, col0 + c - 2, db);
          }
          if (DKV) pp[c >> 1] = pack_bf16x2(p0, p1);
          ds[c >> 1] = pack_bf16x2(g0, g1);
        }
      };
      if (masked) pairs(std::true_type{});
      else pairs(std::false_type{});
      // bf16 pairs over the first 16 columns of this thread's own half (nobody else reads or writes those)
      if (DKV) tmem_st_x16(t_lane + S_COL0 + buf * BW_T + half * HC, pp);
      tmem_st_x16(t_lane + DP_COL0 + buf * BW_T + half * HC, ds);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[buf]);
    }
    // ---- epilogue: accumulators -> bf16 rows in global memory ----
    if (alive && n_steps > 0) {
      if (mbar_wait(acc_full, 0)) {
        tc_fence_after();
      } else {
        give_up(STATUS_TIMEOUT_MBAR);
        alive = false;
      }
    }
    if (alive) {
      const int limit = DKV ? p.sk : p.sq;
      const int o_head = DKV ? kvh : head;
#pragma unroll
      for (int a = 0; a < (DKV ? 2 : 1); ++a) {
        bf16* base = a == 0 ? p.out0 : p.out1;
        const long long sb = a == 0 ? p.o0_sb : p.o1_sb, ss = a == 0 ? p.o0_ss : p.o1_ss, sh = a == 0 ? p.o0_sh : p.o1_sh;
        bf16* orow = base + b * sb + (long long)min(ri, limit - 1) * ss + (long long)o_head * sh + half * HD;
#pragma unroll
        for (int c = 0; c < HD; c += 32) {
          uint32_t o[32];
          if (n_steps > 0) {
            tmem_ld_x32(t_lane + (a == 0 ? ACC0_COL : ACC1_COL) + half * HD + c, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = 0u;
          }
          if (ri < limit) bw_store_row(orow + c, o);
        }
      }
    }
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// The same with 128 streamed rows per step, for head_dim 64 and, without a bias, 128, where step_rows below says so.  Score products of N = 64 (the kernel above) read
// 6 KB of shared memory per 32 clocks of work and leave the tensor core idle between dependent steps; with N = 128 the accumulators and ONE
// buffer of S and of dP fill the 512 columns at head_dim 128, so the two are handed over separately and the products interleave:
//
//   dK / dV:  dV += P^T dO (n) | S^T (n + 1) | dK += dS^T Q (n) | dP^T (n + 1)        elementwise: P (n) | dS (n) | P (n + 1) ...
//   dQ     :  S (n + 1), once S (n) has been read | dQ += dS K (n) | dP (n + 1)
//
// P^T and dS^T overwrite their own scores; every product is issued behind the one that last read its columns.  Sixteen elementwise warps
// (8: 521 against 516 us below).  Streamed tiles arrive through two rings, three tiles of the operand that is needed last (Q or K, with the
// bias) and two of the other.  Shared memory at head_dim 128: 64 KB resident + 160 KB streamed + statistics, which leaves no room for a
// bias.  What bounds it: the chain of a step, S -> P -> dV and dP -> dS -> dK through one buffer each, and fill and drain of a CTA; the tensor pipe is active
// for 47 % (dQ 50 %) of the causal launch below.  (Next would be shared memory: 192 KB read and 64 KB filled per 2048 clocks of dK / dV products.)
// Whole backward, 32 heads of 128: 4 x 2048 causal 558 -> 507 us, 2 x 2080 344 -> 323, without a mask 560 -> 518; 1 x 1000 65.7 -> 61.3.
// Attention layer with relative positions (16 x 512, 32 heads of 64, with the projections) 1473 -> 1434.  Short and ragged sequences: step_rows.
//
// T = 64 is the same with 64 streamed rows, at head_dim 64 and for dQ at 128: half of the tensor-memory columns, registers and shared memory, and two CTAs per
// SM, which fill each other's chains, prologues and epilogues.
template <int D, bool DKV, int T, int BIAS>
struct Bww {
  static constexpr int CTAS = T == 64 ? 2 : 1;
  static constexpr int WARPS = 16 / CTAS;                  // elementwise warps
  static constexpr int THREADS = 64 + 32 * WARPS;
  static constexpr int S1 = T == 64 && (BIAS == 2 || D == 128) ? 2 : 3, S2 = T == 64 && D == 128 ? 1 : 2;  // ring depths: Q (dK / dV) or K (dQ), with the bias; dO or V
  static constexpr int BARS = 1 + 2 * (S1 + S2) + 7;
  static constexpr uint32_t TILE = D / 64 * T * 128;       // one streamed tile
  static constexpr uint32_t BIAS_BYTES = T * BW_R * 2;     // bias elements of one step
  static constexpr size_t STATS = DKV ? 2 * T * sizeof(float2) : 0;
  static constexpr size_t SMEM = size_t(2 * (D / 64)) * FA_BLOCK_BYTES + (S1 + S2) * TILE + (BIAS == 2 ? S1 * BIAS_BYTES : 0) + STATS + BARS * 8 + 16;
  static_assert(CTAS * (SMEM + 1024) <= 228 * 1024, "shared memory of an SM");
};

template <int D, bool DKV, int BIAS, int T>
__global__ void __launch_bounds__(Bww<D, DKV, T, BIAS>::THREADS, Bww<D, DKV, T, BIAS>::CTAS)
attn_bwd_wide_kernel(const __grid_constant__ CUtensorMap tmap_r1, const __grid_constant__ CUtensorMap tmap_r2,
                     const __grid_constant__ CUtensorMap tmap_t1, const __grid_constant__ CUtensorMap tmap_t2,
                     const __grid_constant__ CUtensorMap tmap_b, const BwParams p) {
  using B = Bww<D, DKV, T, BIAS>;
  constexpr int DB = D / 64, BWW_S1 = B::S1, BWW_S2 = B::S2, BWW_WARPS = B::WARPS;
  constexpr uint32_t R_TILE = DB * FA_BLOCK_BYTES, TILE = B::TILE, T_BLOCK = T * 128, BWW_BIAS = B::BIAS_BYTES;
  constexpr uint32_t TMEM_COLS = 512 / B::CTAS, S_COL = 0, DP_COL = T, ACC0_COL = 2 * T, ACC1_COL = ACC0_COL + D;
  constexpr bool RES_TMEM = T == 128 ? !DKV || D == 64 : !DKV && D == 64;  // the resident tiles as tensor-memory operands, where the columns leave room
  constexpr uint32_t RES_COL = ACC0_COL + (DKV ? 2 : 1) * D;
  static_assert(ACC0_COL + (DKV ? 2 : 1) * D <= TMEM_COLS && (!RES_TMEM || RES_COL + D <= TMEM_COLS), "tensor memory columns");
  constexpr uint32_t IDESC_S = make_idesc_bf16(BW_R, T, false, false);
  constexpr uint32_t IDESC_ACC = make_idesc_bf16(BW_R, D, false, true);

  extern __shared__ __align__(1024) uint8_t bww_smem[];
  uint8_t* smem = bww_smem;
  if (smem_u32(smem) & 1023) {  // (the swizzle patterns need it, and there is no room to round up)
    if (threadIdx.x == 0) atomicMax(p.status, STATUS_BAD_ARG);
    return;
  }
  uint8_t* r1_s = smem;
  uint8_t* r2_s = r1_s + R_TILE;
  uint8_t* t1_s = r2_s + R_TILE;            // [BWW_S1]
  uint8_t* t2_s = t1_s + BWW_S1 * TILE;   // [BWW_S2]
  uint8_t* bias_s = t2_s + BWW_S2 * TILE;     // [BWW_S1], BIAS == 2 only
  float* stat_s = reinterpret_cast<float*>(bias_s + (BIAS == 2 ? BWW_S1 * BWW_BIAS : 0));  // dK / dV, [2 steps]: -lse * log2(e) of 128 streamed queries (-inf = no such query), -delta * scale
  uint64_t* bars = reinterpret_cast<uint64_t*>(stat_s + B::STATS / sizeof(float));
  uint64_t* r_full = bars;
  uint64_t* t1_full = bars + 1;
  uint64_t* t1_empty = t1_full + BWW_S1;
  uint64_t* t2_full = t1_empty + BWW_S1;
  uint64_t* t2_empty = t2_full + BWW_S2;
  uint64_t* s_full = t2_empty + BWW_S2;   // S of the step is there
  uint64_t* s_done = s_full + 1;          // dK / dV: P is there (over S); dQ: S has been read
  uint64_t* dp_full = s_done + 1;         // dP of the step is there
  uint64_t* ds_full = dp_full + 1;        // dS is there (over dP)
  uint64_t* acc_full = ds_full + 1;
  uint64_t* res_full = acc_full + 1;      // dQ: the resident tiles are in tensor memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int b = blockIdx.z;
  const int shift = p.sk - p.sq;  // query i may see keys j <= i + shift when causal
  const int group = p.q_heads / p.kv_heads;
  int r0, head, kvh, step0, per_head, n_steps;
  if (DKV) {
    r0 = blockIdx.x * BW_R;
    kvh = blockIdx.y;
    head = kvh * group;
    const int q_steps = (p.sq + T - 1) / T;
    step0 = p.causal ? max(0, r0 - shift) / T : 0;
    per_head = max(0, q_steps - step0);
    n_steps = per_head * group;
  } else {
    r0 = (gridDim.x - 1 - blockIdx.x) * BW_R;
    head = blockIdx.y;
    kvh = head / group;
    int kv_end = p.sk;
    if (p.causal) kv_end = min(p.sk, r0 + BW_R + shift);
    step0 = 0;
    per_head = kv_end > 0 ? (kv_end + T - 1) / T : 0;
    n_steps = per_head;
  }

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_r1);
    prefetch_tmap(&tmap_r2);
    prefetch_tmap(&tmap_t1);
    prefetch_tmap(&tmap_t2);
    mbar_init(r_full, 1);
    for (int s = 0; s < BWW_S1; ++s) {
      mbar_init(&t1_full[s], 1);
      mbar_init(&t1_empty[s], 1);
    }
    for (int s = 0; s < BWW_S2; ++s) {
      mbar_init(&t2_full[s], DKV ? 2 : 1);  // the TMA bytes, and for dK / dV the step's statistics written by the producer warp
      mbar_init(&t2_empty[s], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(s_done, BWW_WARPS);  // one arrival per elementwise warp
    mbar_init(dp_full, 1);
    mbar_init(ds_full, BWW_WARPS);
    mbar_init(acc_full, 1);
    mbar_init(res_full, BWW_WARPS);
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

  auto give_up = [&]() {
    atomicMax(p.status, STATUS_TIMEOUT_MBAR);
    *abort_flag = 1;
  };

  if (warp == 0) {
    // ---------------- TMA producer (the whole warp stays together: all lanes write statistics) ----------------
    auto load = [&](uint8_t* dst, uint32_t block, const CUtensorMap* map, uint64_t* bar, int row, int h) {
#pragma unroll
      for (int d = 0; d < DB; ++d) tma_load_4d(dst + d * block, map, bar, d * 64, row, h, b);
    };
    if (n_steps > 0) {
      if (lane == 0) {
        mbar_expect_tx(r_full, 2 * R_TILE);
        load(r1_s, FA_BLOCK_BYTES, &tmap_r1, r_full, r0, DKV ? kvh : head);
        load(r2_s, FA_BLOCK_BYTES, &tmap_r2, r_full, r0, DKV ? kvh : head);
      }
      int g = 0, local = 0;  // query head of the group (dK / dV), step within it
      for (int n = 0; n < n_steps; ++n) {
        const int s1 = n % BWW_S1, s2 = n % BWW_S2;
        bool ok = !*abort_flag && mbar_wait(&t1_empty[s1], ((n / BWW_S1) & 1) ^ 1);
        const int row0 = (step0 + local) * T;
        const int t_head = DKV ? head + g : kvh;
        if (++local == per_head) { local = 0; ++g; }
        if (ok && lane == 0) {
          mbar_expect_tx(&t1_full[s1], TILE + (BIAS == 2 ? BWW_BIAS : 0));
          load(t1_s + s1 * TILE, T_BLOCK, &tmap_t1, &t1_full[s1], row0, t_head);
          if (BIAS == 2) {
            const int bh = p.b_sh ? (DKV ? t_head : head) : 0, bb = p.b_sb ? b : 0;
            if (DKV) {  // [T queries][128 keys]
              tma_load_4d(bias_s + s1 * BWW_BIAS, &tmap_b, &t1_full[s1], r0, row0, bh, bb);
            } else {  // swizzled blocks of [128 queries][64 keys]
              tma_load_4d(bias_s + s1 * BWW_BIAS, &tmap_b, &t1_full[s1], row0, r0, bh, bb);
              if (T == 128) tma_load_4d(bias_s + s1 * BWW_BIAS + FA_BLOCK_BYTES, &tmap_b, &t1_full[s1], row0 + 64, r0, bh, bb);
            }
          }
        }
        ok = ok && mbar_wait(&t2_empty[s2], ((n / BWW_S2) & 1) ^ 1);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0 && !*abort_flag) give_up();
          break;
        }
        if (lane == 0) {
          mbar_expect_tx(&t2_full[s2], TILE);
          load(t2_s + s2 * TILE, T_BLOCK, &tmap_t2, &t2_full[s2], row0, t_head);
        }
        if (DKV) {
          float2 st[T / 32];
#pragma unroll
          for (int i = 0; i < T / 32; ++i) {
            const int qi = row0 + i * 32 + lane;
            st[i] = make_float2(-INFINITY, 0.f);
            if (qi < p.sq) {
              const long long idx = ((long long)b * p.q_heads + t_head) * p.sq + qi;
              const float l = __ldg(p.lse + idx);
              if (l != -INFINITY) st[i].x = -l * 1.4426950408889634f;  // (a query without a visible key has P = 0 everywhere)
              st[i].y = -__ldg(p.delta + idx) * p.scale;
            }
          }
          // the statistics of step n - 2 are read until its dS is there, which the release of its Q tile tells
          ok = n < 2 || mbar_wait(&t1_empty[(n - 2) % BWW_S1], ((n - 2) / BWW_S1) & 1);
          if (!__all_sync(0xffffffffu, ok)) {
            if (lane == 0 && !*abort_flag) give_up();
            break;
          }
#pragma unroll
          for (int i = 0; i < T / 32; ++i) {
            stat_s[s2 * 2 * T + i * 32 + lane] = st[i].x;
            stat_s[(s2 * 2 + 1) * T + i * 32 + lane] = st[i].y;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&t2_full[s2]);
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the warp stays together, one lane issues: see umma_bf16_lead) ----------------
    if (n_steps > 0) {
      const uint32_t leader = elect_one();
      const uint32_t r1_lo = desc_kmajor_lo(smem_u32(r1_s)), r2_lo = desc_kmajor_lo(smem_u32(r2_s));
      auto scores = [&](int which, uint32_t tile) {  // S = R1 T1^T (0) or dP = R2 T2^T (1)
        const uint32_t t_lo = desc_kmajor_lo(tile), col = tmem_base + (which ? DP_COL : S_COL);
#pragma unroll
        for (int d = 0; d < DB; ++d) {
#pragma unroll
          for (int kk = 0; kk < 64 / 16; ++kk) {
            const uint32_t off = d * (T_BLOCK >> 4) + kk * 2;
            if (!RES_TMEM) umma_bf16_lead(leader, col, (which ? r2_lo : r1_lo) + d * (FA_BLOCK_BYTES >> 4) + kk * 2, t_lo + off, IDESC_S, (d | kk) ? 1u : 0u);
            else umma_bf16_tmem_a_lead(leader, col, tmem_base + RES_COL + which * (D / 2) + (d * 4 + kk) * 8, t_lo + off, IDESC_S, (d | kk) ? 1u : 0u);
          }
        }
        umma_commit_lead(leader, which ? dp_full : s_full);
      };
      // dQ reads its V tile in dP only (dO is read again, in dV).  Two CTAs per SM, with their short rings, free it at once (head_dim 64, 2 x 4096, 16 heads:
      // whole backward 500 -> 496 us); with one CTA the extra commit in the middle of a step's chain costs more (head_dim 128, causal: 441 -> 444 us).
      auto dp_scores = [&](int n) {
        scores(1, smem_u32(t2_s + (n % BWW_S2) * TILE));
        if (!DKV && T == 64) umma_commit_lead(leader, &t2_empty[n % BWW_S2]);
      };
      auto accumulate = [&](uint32_t acc_col, uint32_t a_col, uint32_t tile, bool first) {
        const uint32_t t_lo = desc_mnmajor_lo(tile, T_BLOCK);
#pragma unroll
        for (int kk = 0; kk < T / 16; ++kk)  // (the bf16 operand of 32 streamed rows lies in the first half of their own columns)
          umma_bf16_tmem_a_lead(leader, tmem_base + acc_col, tmem_base + a_col + (kk >> 1) * 32 + (kk & 1) * 8, t_lo + kk * (16 * 128 >> 4), IDESC_ACC,
                                (!first || kk) ? 1u : 0u);
      };
      auto wait_all = [&](uint64_t* bar, uint32_t parity) {
        const bool there = __all_sync(0xffffffffu, mbar_wait(bar, parity));
        if (!there && leader) give_up();
        tc_fence_after();
        return there;
      };
      auto t1_at = [&](int n) { return smem_u32(t1_s + (n % BWW_S1) * TILE); };
      auto t2_at = [&](int n) { return smem_u32(t2_s + (n % BWW_S2) * TILE); };
      auto t1_there = [&](int n) { return wait_all(&t1_full[n % BWW_S1], (n / BWW_S1) & 1); };
      auto t2_there = [&](int n) { return wait_all(&t2_full[n % BWW_S2], (n / BWW_S2) & 1); };
      bool ok = wait_all(RES_TMEM ? res_full : r_full, 0) && t1_there(0);
      if (ok) scores(0, t1_at(0));
      ok = ok && t2_there(0);
      if (ok) dp_scores(0);
      for (int n = 0; ok && n < n_steps; ++n) {
        const bool more = n + 1 < n_steps;
        ok = wait_all(s_done, n & 1);
        if (!ok) break;
        if (DKV) {
          accumulate(ACC1_COL, S_COL, t2_at(n), n == 0);
          umma_commit_lead(leader, &t2_empty[n % BWW_S2]);  // (dP^T of this step has read dO before)
        }
        if (more) {
          ok = t1_there(n + 1);
          if (!ok) break;
          scores(0, t1_at(n + 1));
        }
        ok = wait_all(ds_full, n & 1);
        if (!ok) break;
        accumulate(ACC0_COL, DP_COL, t1_at(n), n == 0);
        umma_commit_lead(leader, &t1_empty[n % BWW_S1]);
        if (!DKV && T == 128) umma_commit_lead(leader, &t2_empty[n % BWW_S2]);
        if (more) {
          ok = t2_there(n + 1);
          if (!ok) break;
          dp_scores(n + 1);
        }
      }
      umma_commit_lead(leader, acc_full);
    }
  } else {
    // ---------------- elementwise warps: two or four threads per TMEM lane, 32 of the step's columns each ----------------
    constexpr int HC = T / (BWW_WARPS / 4), HD = D / (BWW_WARPS / 4);
    static_assert(HC == 32, "columns per thread");
    const int quarter = warp & 3;  // TMEM lane quarter this warp may access
    const int part = (warp - 2) >> 2;
    const int row = quarter * 32 + lane;
    const int ri = r0 + row;  // key (DKV) or query
    const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16);
    float my_lse2 = -INFINITY, my_del = 0.f;  // negated
    if (!DKV && ri < p.sq) {
      const long long idx = ((long long)b * p.q_heads + head) * p.sq + ri;
      const float l = __ldg(p.lse + idx);
      if (l != -INFINITY) my_lse2 = -l * 1.4426950408889634f;
      my_del = -__ldg(p.delta + idx) * p.scale;
    }
    bool alive = true;
    int g = 0, local = 0;  // as in the producer
    if (RES_TMEM && n_steps > 0) {
      // resident tiles: swizzled shared memory -> tensor memory, half a row of one tile per thread
      if (!mbar_wait(r_full, 0)) {
        give_up();
        alive = false;
      }
      if (part < 2 * DB) {
        const uint8_t* block = (part / DB ? r2_s : r1_s) + (part % DB) * FA_BLOCK_BYTES;
        uint32_t w[32];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint4 u = *reinterpret_cast<const uint4*>(block + row * 128 + ((c ^ (row & 7)) << 4));
          w[4 * c] = u.x; w[4 * c + 1] = u.y; w[4 * c + 2] = u.z; w[4 * c + 3] = u.w;
        }
        __syncwarp();
        tmem_st_x32(t_lane + RES_COL + part * 32, w);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(res_full);
    }
    // every lane learns whether all lanes of its warp saw the barrier complete
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
      const bool there = __all_sync(0xffffffffu, !*abort_flag && mbar_wait(bar, parity));
      if (!there) {
        if (lane == 0 && !*abort_flag) give_up();
        alive = false;
      }
      return there;
    };

    for (int n = 0; alive && n < n_steps; ++n) {
      const float* neg_lse = stat_s + (n % BWW_S2) * 2 * T + part * HC;
      const float* neg_delta = neg_lse + T;
      if (DKV && !wait_all(&t2_full[n % BWW_S2], (n / BWW_S2) & 1)) break;
      if (BIAS == 2 && !wait_all(&t1_full[n % BWW_S1], (n / BWW_S1) & 1)) break;
      if (!wait_all(s_full, n & 1)) break;
      tc_fence_after();
      const int col0 = (step0 + local) * T + part * HC;  // first query (DKV) or key of my columns
      const int b_head = DKV ? head + g : head;
      if (++local == per_head) { local = 0; ++g; }
      // score bias: element (query, key) = (col0 + c, ri) for dK / dV - there the lanes of a warp own consecutive keys - and
      // (ri, col0 + c) for dQ, where a thread's columns are consecutive keys of one row and are read eight at a time
      const long long bias_base = BIAS ? (long long)b * p.b_sb + (long long)b_head * p.b_sh + (long long)ri * (DKV ? p.b_sk : p.b_sq) : 0;
      const long long bias_step = DKV ? p.b_sq : p.b_sk;  // per column
      const int col_limit = DKV ? p.sq : p.sk, row_limit = DKV ? p.sk : p.sq;
      // ---- P = exp(S * scale - lse) ----
      float pr[HC], bv[8];
      {
        uint32_t sv[HC];
        tmem_ld_x32(t_lane + S_COL + part * HC, sv);
        tmem_ld_wait();
        if (!DKV) {  // S may be overwritten
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_done);
        }
        const uint32_t visible = bw_visible<DKV>(p, ri, shift, col0);
        const bool masked = __any_sync(0xffffffffu, visible != 0xffffffffu);  // (per warp)
#pragma unroll
        for (int c = 0; c < HC; c += 4) {
          const float4 l = DKV ? *reinterpret_cast<const float4*>(neg_lse + c) : make_float4(my_lse2, my_lse2, my_lse2, my_lse2);
          if (BIAS && (c & 7) == 0) {
            if (BIAS == 1) {
              load_bias8(p.bias, p.bias_kind, bias_base + (long long)(col0 + c) * bias_step, bias_step, ri < row_limit ? col_limit - col0 - c : 0,
                         !DKV && p.bias_vec, bv);
            } else {
              bw_bias8<DKV>(bias_s + (n % BWW_S1) * BWW_BIAS, row, part * HC + c, bv);
            }
          }
          float x0, x1, x2, x3;
          ffma2(x0, x1, __uint_as_float(sv[c]), __uint_as_float(sv[c + 1]), p.scale_log2e, p.scale_log2e, l.x, l.y);
          ffma2(x2, x3, __uint_as_float(sv[c + 2]), __uint_as_float(sv[c + 3]), p.scale_log2e, p.scale_log2e, l.z, l.w);
          if (BIAS) {
            constexpr float LOG2E = 1.4426950408889634f;
            ffma2(x0, x1, bv[c & 7], bv[(c & 7) + 1], LOG2E, LOG2E, x0, x1);
            ffma2(x2, x3, bv[(c & 7) + 2], bv[(c & 7) + 3], LOG2E, LOG2E, x2, x3);
          }
          pr[c] = ex2_approx(x0);
          pr[c + 1] = ex2_approx(x1);
          pr[c + 2] = ex2_approx(x2);
          pr[c + 3] = ex2_approx(x3);
        }
        if (masked) {
#pragma unroll
          for (int c = 0; c < HC; ++c)
            if (!(visible >> c & 1)) pr[c] = 0.f;
        }
      }
      uint32_t packed[HC / 2];
      if (DKV) {  // bf16 pairs over the first half of this thread's own columns (nobody else reads or writes those)
#pragma unroll
        for (int c = 0; c < HC; c += 2) packed[c >> 1] = pack_bf16x2(pr[c], pr[c + 1]);
        tmem_st_x16(t_lane + S_COL + part * HC, packed);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(s_done);
      }
      // ---- dS = P * (dP - delta) * scale ----
      if (!wait_all(dp_full, n & 1)) break;
      tc_fence_after();
      uint32_t dv[HC];
      tmem_ld_x32(t_lane + DP_COL + part * HC, dv);
      tmem_ld_wait();
#pragma unroll
      for (int c = 0; c < HC; c += 4) {
        const float4 d = DKV ? *reinterpret_cast<const float4*>(neg_delta + c) : make_float4(my_del, my_del, my_del, my_del);
        float g0, g1, g2, g3;
        ffma2(g0, g1, __uint_as_float(dv[c]), __uint_as_float(dv[c + 1]), p.scale, p.scale, d.x, d.y);
        ffma2(g2, g3, __uint_as_float(dv[c + 2]), __uint_as_float(dv[c + 3]), p.scale, p.scale, d.z, d.w);
        ffma2(g0, g1, g0, g1, pr[c], pr[c + 1], 0.f, 0.f);
        ffma2(g2, g3, g2, g3, pr[c + 2], pr[c + 3], 0.f, 0.f);
        if (BIAS && !DKV && p.dbias && ri < row_limit) {
          // d(bias) = P (dP - delta) = dS / scale; pairs that are masked or out of range contribute nothing
          const float db[4] = {pr[c] != 0.f ? g0 * p.inv_scale : 0.f, pr[c + 1] != 0.f ? g1 * p.inv_scale : 0.f, pr[c + 2] != 0.f ? g2 * p.inv_scale : 0.f,
                               pr[c + 3] != 0.f ? g3 * p.inv_scale : 0.f};
          bw_add_dbias(p, bias_base, col0 + c, db);
        }
        packed[c >> 1] = pack_bf16x2(g0, g1);
        packed[(c >> 1) + 1] = pack_bf16x2(g2, g3);
      }
      tmem_st_x16(t_lane + DP_COL + part * HC, packed);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_full);
    }
    // ---- epilogue: accumulators -> bf16 rows in global memory ----
    if (alive && n_steps > 0 && wait_all(acc_full, 0)) tc_fence_after();
    if (alive) {
      const int limit = DKV ? p.sk : p.sq;
      const int o_head = DKV ? kvh : head;
#pragma unroll
      for (int a = 0; a < (DKV ? 2 : 1); ++a) {
        bf16* base = a == 0 ? p.out0 : p.out1;
        const long long sb = a == 0 ? p.o0_sb : p.o1_sb, ss = a == 0 ? p.o0_ss : p.o1_ss, sh = a == 0 ? p.o0_sh : p.o1_sh;
        bf16* orow = base + b * sb + (long long)min(ri, limit - 1) * ss + (long long)o_head * sh + part * HD;
        constexpr int W = HD < 32 ? HD : 32;
#pragma unroll
        for (int c = 0; c < HD; c += W) {
          uint32_t o[W];
          if (n_steps > 0) {
            __syncwarp();
            const uint32_t at = t_lane + (a == 0 ? ACC0_COL : ACC1_COL) + part * HD + c;
            if constexpr (W == 32) tmem_ld_x32(at, o);
            else tmem_ld_x16(at, o);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int i = 0; i < W; ++i) o[i] = 0u;
          }
          if (ri < limit) bw_store_row(orow + c, o);
        }
      }
    }
  }

  // ---------------- teardown ----------------
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// ---- gradient of a bias that several (batch, head) pairs share ----
//
// d(bias)[i, j] = sum over the pairs of P (dP - delta).  Inside the dQ launch every pair adds its own 4 bytes per score into one fp32 buffer: 134 M
// reductions for 16 x 512 tokens and 32 heads, 126 us of its 235.  Here a CTA owns a tile of 128 queries x 64 keys of the bias and walks the pairs:
// S = Q K^T and dP = dO V^T once more (seven tile products become nine), the sum of P (dP - delta) in registers, one store at the end and no
// buffer to clear.  Sums run in a fixed order.
//
//   warp 0    : TMA producer, the four tiles of a pair (Q, dO, K, V) per stage of a ring
//   warp 1    : MMA issuer, S and dP of pair n + 1 while the other warps are at pair n (two buffers of each: 256 TMEM columns)
//   warps 2-9 : two threads per query, 32 keys each, their sums in registers, their biases (the same for every pair) in slots of their own in
//               shared memory
//
// Two CTAs per SM.  One with tiles of 128 keys, sixteen such warps and a third less to load took 110 us for that shape (2000 clocks per tile and pair, half of them an
// exponential per score on the special-function unit, the rest latencies of barrier and TMEM that warps in step do not hide from each other); this one
// takes 88 us.  Whole backward with it 307 us, with reductions in the dQ launch, the buffer to clear and the cast to bf16 353.  Where it pays: ops/native.py.
constexpr int BG_STAGES = 2, BG_KEYS = 64, BG_WARPS = 8, BG_THREADS = 64 + 32 * BG_WARPS;
constexpr size_t BG_SMEM = size_t(BG_STAGES) * 2 * (FA_BLOCK_BYTES + BG_KEYS * 128) + BW_R * BG_KEYS * 2 + 16 * 8;
static_assert(2 * (BG_SMEM + 1024) <= 228 * 1024, "shared memory of an SM");

struct BgParams {
  int batch, sq, sk, q_heads, kv_heads, causal;
  float scale_log2e;
  const float *lse, *delta;  // [batch][q_heads][sq]
  const bf16* bias;          // element strides over (head, query), keys contiguous; b_sh = 0: shared by the heads too
  void* dbias;               // in the bias' own strides
  int dbias_fp32;
  long long b_sh, b_sq;
  uint32_t* status;
};

__global__ void __launch_bounds__(BG_THREADS, 2)
attn_bias_grad_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_do, const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const BgParams p) {
  constexpr uint32_t TILE = FA_BLOCK_BYTES, K_TILE = BG_KEYS * 128, STAGE = 2 * (TILE + K_TILE);  // Q, dO, K, V of one pair, head_dim 64
  constexpr uint32_t TMEM_COLS = 256;
  constexpr uint32_t IDESC_S = make_idesc_bf16(BW_R, BG_KEYS, false, false);
  extern __shared__ __align__(1024) uint8_t bg_smem[];
  uint8_t* smem = bg_smem;
  if (smem_u32(smem) & 1023) {  // (the swizzle patterns need it, and there is no room to round up)
    if (threadIdx.x == 0) atomicMax(p.status, STATUS_BAD_ARG);
    return;
  }
  uint4* bias_s = reinterpret_cast<uint4*>(smem + BG_STAGES * STAGE);  // [4 chunks of 8 keys][threads], private
  uint64_t* t_full = reinterpret_cast<uint64_t*>(bias_s + 4 * 32 * BG_WARPS);
  uint64_t* t_empty = t_full + BG_STAGES;
  uint64_t* s_full = t_empty + BG_STAGES;  // [2 buffers]: S and dP of a pair are there
  uint64_t* s_done = s_full + 2;           // and have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(s_done + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int k0 = blockIdx.x * BG_KEYS, q0 = blockIdx.y * BW_R, plane = blockIdx.z;
  const int shift = p.sk - p.sq, group = p.q_heads / p.kv_heads;
  const int heads = p.b_sh ? 1 : p.q_heads;  // heads that share the plane
  const bool any = !p.causal || k0 <= min(p.sq, q0 + BW_R) - 1 + shift;  // (otherwise no query of the tile sees a key of it)
  const int pairs = any ? p.batch * heads : 0;

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_q);
    prefetch_tmap(&tmap_do);
    prefetch_tmap(&tmap_k);
    prefetch_tmap(&tmap_v);
    for (int s = 0; s < BG_STAGES; ++s) {
      mbar_init(&t_full[s], 1);
      mbar_init(&t_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_done[s], BG_WARPS);
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
  auto give_up = [&]() {
    atomicMax(p.status, STATUS_TIMEOUT_MBAR);
    *abort_flag = 1;
  };

  if (warp == 0) {
    if (lane == 0) {
      for (int n = 0, b = 0, h = plane; n < pairs; ++n) {
        const int s = n % BG_STAGES;
        if (*abort_flag || !mbar_wait(&t_empty[s], ((n / BG_STAGES) & 1) ^ 1)) {
          if (!*abort_flag) give_up();
          break;
        }
        uint8_t* dst = smem + s * STAGE;
        mbar_expect_tx(&t_full[s], STAGE);
        tma_load_4d(dst, &tmap_q, &t_full[s], 0, q0, h, b);
        tma_load_4d(dst + 2 * TILE, &tmap_k, &t_full[s], 0, k0, h / group, b);
        tma_load_4d(dst + TILE, &tmap_do, &t_full[s], 0, q0, h, b);
        tma_load_4d(dst + 2 * TILE + K_TILE, &tmap_v, &t_full[s], 0, k0, h / group, b);
        if (heads > 1 && ++h < heads) continue;
        if (heads > 1) h = 0;
        ++b;
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = elect_one();
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
      const bool there = __all_sync(0xffffffffu, !*abort_flag && mbar_wait(bar, parity));
      if (!there && leader && !*abort_flag) give_up();
      tc_fence_after();
      return there;
    };
    for (int n = 0; n < pairs; ++n) {
      const int s = n % BG_STAGES, buf = n & 1;
      if (!wait_all(&t_full[s], (n / BG_STAGES) & 1)) break;
      if (n >= 2 && !wait_all(&s_done[buf], ((n >> 1) & 1) ^ 1)) break;
      const uint32_t at = smem_u32(smem + s * STAGE);
#pragma unroll
      for (int which = 0; which < 2; ++which) {
        const uint32_t a_lo = desc_kmajor_lo(at + which * TILE), b_lo = desc_kmajor_lo(at + 2 * TILE + which * K_TILE);
#pragma unroll
        for (int i = 0; i < 4; ++i) umma_bf16_lead(leader, tmem_base + (buf * 2 + which) * BG_KEYS, a_lo + i * 2, b_lo + i * 2, IDESC_S, i ? 1u : 0u);
      }
      umma_commit_lead(leader, &s_full[buf]);
      umma_commit_lead(leader, &t_empty[s]);
    }
  } else {
    constexpr int HC = BG_KEYS / (BG_WARPS / 4);
    static_assert(HC == 32, "keys per thread");
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    const int ri = q0 + quarter * 32 + lane, col0 = k0 + part * HC;
    const uint32_t t_lane = tmem_base + (uint32_t(quarter * 32) << 16) + part * HC;
    const bool row_ok = ri < p.sq;
    const long long row_at = plane * p.b_sh + (long long)ri * p.b_sq + col0;
    const uint32_t visible = row_ok ? bw_bits(0, min(p.sk, p.causal ? ri + shift + 1 : p.sk) - col0) : 0u;
    const bool masked = __any_sync(0xffffffffu, visible != 0xffffffffu);  // (per warp)
    uint4* my_bias = bias_s + threadIdx.x - 64;
#pragma unroll
    for (int c = 0; c < HC; c += 8) {
      uint4 u = make_uint4(0, 0, 0, 0);
      if (row_ok && col0 + c + 8 <= p.sk) {
        u = __ldg(reinterpret_cast<const uint4*>(p.bias + row_at + c));
      } else if (row_ok) {
        uint32_t* w = &u.x;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (col0 + c + i < p.sk) w[i >> 1] |= uint32_t(__bfloat16_as_ushort(p.bias[row_at + c + i])) << (16 * (i & 1));
      }
      my_bias[c / 8 * (32 * BG_WARPS)] = u;
    }
    float acc[HC];
#pragma unroll
    for (int c = 0; c < HC; ++c) acc[c] = 0.f;
    // my row of the pairs' statistics: the pairs are batches (one head's plane) or all heads of all batches, one [sq] row apart or q_heads of them
    const long long stat_step = heads > 1 ? p.sq : (long long)p.q_heads * p.sq;
    const float *lse_at = p.lse + (long long)plane * p.sq + ri, *delta_at = p.delta + (long long)plane * p.sq + ri;
    float l2 = -INFINITY, del = 0.f;  // -lse * log2(e) (-inf: no such query, or none of its keys visible) and -delta
    auto stats = [&]() {
      const float l = __ldg(lse_at);
      l2 = l != -INFINITY ? -l * 1.4426950408889634f : -INFINITY;
      del = -__ldg(delta_at);
      lse_at += stat_step;
      delta_at += stat_step;
    };
    if (row_ok && pairs > 0) stats();
    bool alive = true;
    for (int n = 0; n < pairs; ++n) {
      const int buf = n & 1;
      const float l2_now = l2, del_now = del;
      if (row_ok && n + 1 < pairs) stats();
      if (!__all_sync(0xffffffffu, !*abort_flag && mbar_wait(&s_full[buf], (n >> 1) & 1))) {
        if (lane == 0 && !*abort_flag) give_up();
        alive = false;
        break;
      }
      tc_fence_after();
#pragma unroll
      for (int c0 = 0; c0 < HC; c0 += 16) {
        uint32_t sv[16], dv[16];
        tmem_ld_x16(t_lane + buf * 2 * BG_KEYS + c0, sv);
        tmem_ld_x16(t_lane + (buf * 2 + 1) * BG_KEYS + c0, dv);
        const uint4 u0 = my_bias[(c0 / 8) * (32 * BG_WARPS)], u1 = my_bias[(c0 / 8 + 1) * (32 * BG_WARPS)];
        const uint32_t bw[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};  // bf16 pairs
        tmem_ld_wait();
        if (c0 + 16 == HC) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&s_done[buf]);
        }
        float odd0 = 0.f, odd1 = 0.f;  // not 0 if a dP is not finite
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
          constexpr float LOG2E = 1.4426950408889634f;
          const uint32_t w = bw[c / 2];
          float x0, x1, g0, g1;
          ffma2(x0, x1, __uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u), LOG2E, LOG2E, l2_now, l2_now);
          ffma2(x0, x1, __uint_as_float(sv[c]), __uint_as_float(sv[c + 1]), p.scale_log2e, p.scale_log2e, x0, x1);
          sv[c] = __float_as_uint(ex2_approx(x0));
          sv[c + 1] = __float_as_uint(ex2_approx(x1));
          fadd2(g0, g1, __uint_as_float(dv[c]), __uint_as_float(dv[c + 1]), del_now, del_now);
          dv[c] = __float_as_uint(g0);
          dv[c + 1] = __float_as_uint(g1);
          ffma2(odd0, odd1, g0, g1, 0.f, 0.f, odd0, odd1);
        }
        // pairs of a query and a key that are out of range or masked contribute nothing, whatever their dP is
        if (masked) {
#pragma unroll
          for (int c = 0; c < 16; ++c)
            if (!(visible >> (c0 + c) & 1)) sv[c] = 0u;
        }
        if (odd0 + odd1 != 0.f) {
#pragma unroll
          for (int c = 0; c < 16; ++c)
            if (sv[c] == 0u) dv[c] = 0u;
        }
#pragma unroll
        for (int c = 0; c < 16; c += 2)
          ffma2(acc[c0 + c], acc[c0 + c + 1], __uint_as_float(sv[c]), __uint_as_float(sv[c + 1]), __uint_as_float(dv[c]), __uint_as_float(dv[c + 1]), acc[c0 + c],
                acc[c0 + c + 1]);
      }
    }
    if (alive && row_ok) {
#pragma unroll
      for (int c = 0; c < HC; c += 8) {
        if (col0 + c + 8 <= p.sk) {
          if (p.dbias_fp32) {
            float4* dst = reinterpret_cast<float4*>(static_cast<float*>(p.dbias) + row_at + c);
            dst[0] = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
            dst[1] = make_float4(acc[c + 4], acc[c + 5], acc[c + 6], acc[c + 7]);
          } else {
            *reinterpret_cast<uint4*>(static_cast<bf16*>(p.dbias) + row_at + c) =
                make_uint4(pack_bf16x2(acc[c], acc[c + 1]), pack_bf16x2(acc[c + 2], acc[c + 3]), pack_bf16x2(acc[c + 4], acc[c + 5]), pack_bf16x2(acc[c + 6], acc[c + 7]));
          }
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (col0 + c + i >= p.sk) continue;
            if (p.dbias_fp32) static_cast<float*>(p.dbias)[row_at + c + i] = acc[c + i];
            else static_cast<bf16*>(p.dbias)[row_at + c + i] = __float2bfloat16(acc[c + i]);
          }
        }
      }
    }
  }

  // ---------------- teardown ----------------
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

template <int D, bool DKV, int BIAS, int T>
static int bw_launch_wide(const CUtensorMap& r1, const CUtensorMap& r2, const CUtensorMap& t1, const CUtensorMap& t2, const CUtensorMap& tb,
                          const BwParams& p, dim3 grid, cudaStream_t stream) {
  constexpr size_t smem = Bww<D, DKV, T, BIAS>::SMEM;
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TPB_ERR_CUDA;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(attn_bwd_wide_kernel<D, DKV, BIAS, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)
      return TPB_ERR_CUDA;
    configured[dev].store(true, std::memory_order_release);
  }
  attn_bwd_wide_kernel<D, DKV, BIAS, T><<<grid, Bww<D, DKV, T, BIAS>::THREADS, smem, stream>>>(r1, r2, t1, t2, tb, p);
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

template <int D, bool DKV, int BIAS>
static int bw_launch(const CUtensorMap& r1, const CUtensorMap& r2, const CUtensorMap& t1, const CUtensorMap& t2, const CUtensorMap& tb, const BwParams& p,
                     dim3 grid, cudaStream_t stream) {
  constexpr size_t smem = size_t(D / 64) * (2 * FA_BLOCK_BYTES + 2 * BW_STAGES * BW_T_BLOCK_BYTES) + (BIAS == 2 ? BW_STAGES * BW_BIAS_BYTES : 0) +
                          2 * BW_STAGES * BW_T * sizeof(float) + 1024 + 256;
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TPB_ERR_CUDA;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(attn_bwd_tcgen05_kernel<D, DKV, BIAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess)
      return TPB_ERR_CUDA;
    configured[dev].store(true, std::memory_order_release);
  }
  attn_bwd_tcgen05_kernel<D, DKV, BIAS><<<grid, BW_THREADS, smem, stream>>>(r1, r2, t1, t2, tb, p);
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}

// Streamed rows per step of a launch with one CTA per SM, 64 or 128: which kernel it takes.  bias_mode as BIAS above; heads: of the launch's grid (KV heads for
// dK / dV).  What decides is how many rows of the last step are empty, in every product and elementwise pass, against what a step costs.
// Times are of whole backwards, both launches in steps of 64 / of 128 rows, in us, causal where no bias is named.
//   head_dim 128 with a bias: 64, the wide rings leave no room for it.
//   head_dim 128: 64 for a sequence that ends in the first half of its first, second or third wide step (32 heads: 1 x 33 12.2 / 13.4, 8 x 150
//   52.7 / 54.8, 2 x 300 32.0 / 33.2); from the fourth on wide steps win all the same (2 x 420 41.9 / 41.2, 4 x 700 133 / 128).
//   head_dim 64, the same line (32 heads: 4 x 33 12.5 / 14.8, 8 x 150 38.6 / 44.4, 8 x 300 65.4 / 73.3), and with 64 heads x batches and more, several
//   rounds of CTAs, up to the fifth (32 heads: 2 x 420 33.9 / 34.8, 16 x 420 191 / 202, 2 x 576 3 % and
//   1 x 576 -4 %; 4 x 420, 12 heads 33.5 / 30.9).  At six steps either may be 3 % ahead.
//   head_dim 64, one or two whole steps of very many heads: the smaller CTA's shorter fill and drain, many times over (32 heads: 16 x 100 38.6 / 40.9, 4 x 100 14.2 / 14.2).
//   head_dim 64 with a bias: 64 only for up to 64 rows (32 heads: 4 x 64 10 %, with a padding mask 7 % longer in wide steps); beyond, the wide
//   kernel's warps, twice as many per bias element, decide (4 x 300 0.79 of the time, 2 x 900 0.71, with a mask 0.76 and 0.64).
static int step_rows(int head_dim, int bias_mode, int streamed, int heads, int batch) {
  const bool half = streamed % 128 > 0 && streamed % 128 <= BW_T;
  if (head_dim == 128) return bias_mode || (half && streamed < 3 * 128) ? BW_T : 128;
  if (bias_mode) return streamed <= BW_T ? BW_T : 128;
  const long long rows = (long long)heads * batch;
  if (half) return streamed < 3 * 128 || (streamed < 5 * 128 && rows >= 64) ? BW_T : 128;
  return streamed <= 2 * 128 && rows >= 256 ? BW_T : 128;
}

// Whether a launch over `resident` rows takes the wide kernel with two CTAs per SM and steps of 64 rows (head_dim 64): where there are CTAs for it; causal
// CTAs differ in length, so that it takes a second round of them.  Whole backwards in us, as step_rows has it / with two CTAs per SM: 16 x 512, 32 heads
// 256 / 187, causal 209 / 156, with a bias 278 / 219; 4 x 2048, 12 heads 263 / 225, causal 168 / 157; 32 x 129, 16 heads 72 / 55; 4 x 300, 16 heads (192 CTAs)
// 30.3 / 24.8, causal with a mask 46.5 / 49.1; 2 x 1000, 12 heads (192) 54.6 / 48.5, causal 42.6 / 45.9; 1 x 512, 8 heads (32) 20.6 / 23.0.
static bool two_per_sm(int head_dim, int resident, int heads, int batch, bool causal) {
  return head_dim == 64 && (long long)((resident + BW_R - 1) / BW_R) * heads * batch > (causal ? 296 : 148);
}

// The dQ launch at head_dim 128, whose resident tiles and rings of steps of 64 keys just fit half of an SM (with them in shared memory and not in tensor memory, an
// MMA reads twice as much): for sequences of a few steps, whose fill and drain count.  Whole backwards in us, 32 heads, wide / so: 16 x 512 336 / 321, causal 292 / 269;
// 16 x 100 57.2 / 49.3; 3 x 200 33.8 / 30.9; 16 heads 4 x 300 37.3 / 34.6, 2 x 700 55.9 / 52.6, causal 45.3 / 45.5; but 1 x 2048 219 / 222, causal 153 / 163, 4 x 2048 causal 505 / 510.
// From 641 to 1152 keys either is ahead by up to 5 % (2 x 768, 16 heads 55.5 / 53.7, causal 44.9 / 46.6; 4 x 1024, 32 heads 242 / 250, causal 194 / 184), from
// 1280 on wide steps in most (4 x 1536, 32 heads 499 / 563, 2 x 2048 422 / 462, causal 266 / 300), so the line stays where the gain ends.
static bool dq_two_per_sm_128(int head_dim, int sq, int sk, int heads, int batch) {
  return head_dim == 128 && sk <= 640 && (long long)((sq + BW_R - 1) / BW_R) * heads * batch > 148;
}

}  // namespace tpb

using namespace tpb;

// Rows per step (64 or 128) of a launch of tpb_attn_backward_sm100 that streams `streamed` rows; bias: 0 none, 1 element by element, 2 by TMA.
extern "C" int tpb_attn_backward_step_rows(int head_dim, int bias, int streamed, int heads, int batch) { return step_rows(head_dim, bias, streamed, heads, batch); }

// Same contract as tpb_attn_backward_bias (strides in elements, head_dim contiguous; bias strides of 0 broadcast; dbias is fp32 with
// the bias' strides, zero-initialised; `delta` is a [batch][q_heads][sq] fp32
// scratch buffer this call fills) plus: every stride of q / k / v / dout must be a multiple of 8 elements and their bases
// 16-byte aligned (TMA); `status` is a device word that receives a non-zero code if a wait inside a kernel ran out of time.
extern "C" int tpb_attn_backward_sm100(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                                       float* delta, void* dq, void* dk, void* dv, int batch, int sq, int sk, int q_heads, int kv_heads,
                                       int head_dim, long long q_sb, long long q_ss, long long q_sh, long long k_sb, long long k_ss,
                                       long long k_sh, long long v_sb, long long v_ss, long long v_sh, long long o_sb, long long o_ss,
                                       long long o_sh, long long do_sb, long long do_ss, long long do_sh, long long dq_sb, long long dq_ss,
                                       long long dq_sh, long long dk_sb, long long dk_ss, long long dk_sh, int causal, float scale,
                                       const void* bias, int bias_dtype, long long bias_sb, long long bias_sh, long long bias_sq,
                                       long long bias_sk, float* dbias, void* status, void* stream_) {
  if (!q || !k || !v || !out || !dout || !lse || !delta || !dq || !dk || !dv || !status || batch <= 0 || sq <= 0 || sk <= 0 || q_heads <= 0 ||
      kv_heads <= 0 || q_heads % kv_heads)
    return TPB_ERR_ARG;
  if (head_dim != 64 && head_dim != 128) return TPB_ERR_SIZE;
  if ((bias && bias_dtype != 0 && bias_dtype != 1) || (dbias && !bias) || (bias && !(scale > 0.f))) return TPB_ERR_ARG;
  const long long strides[] = {q_ss, k_ss, v_ss, do_ss, q_heads > 1 ? q_sh : 0, q_heads > 1 ? do_sh : 0, kv_heads > 1 ? k_sh : 0,
                               kv_heads > 1 ? v_sh : 0, batch > 1 ? q_sb : 0, batch > 1 ? k_sb : 0, batch > 1 ? v_sb : 0, batch > 1 ? do_sb : 0};
  for (long long s : strides)
    if (s & 7) return TPB_ERR_ALIGN;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)dout) & 15) return TPB_ERR_ALIGN;
  if ((dq_ss | dq_sh | dq_sb | dk_ss | dk_sh | dk_sb) & 1 || (((uintptr_t)dq | (uintptr_t)dk | (uintptr_t)dv) & 3)) return TPB_ERR_ALIGN;
  if (fa_bind_thread() != TPB_OK) return TPB_ERR_CUDA;
  cudaStream_t s = static_cast<cudaStream_t>(stream_);
  int rc = tpb_attn_bwd_delta(out, dout, delta, batch, sq, q_heads, head_dim, o_sb, o_ss, o_sh, do_sb, do_ss, do_sh, stream_);
  if (rc != TPB_OK) return rc;
  CUtensorMap q128, do128, k128, v128, q64, do64, k64, v64;
  rc = fa_tmap(&q128, q, head_dim, BW_R, sq, q_heads, batch, q_ss, q_sh, q_sb);
  if (rc == TPB_OK) rc = fa_tmap(&do128, dout, head_dim, BW_R, sq, q_heads, batch, do_ss, do_sh, do_sb);
  if (rc == TPB_OK) rc = fa_tmap(&k128, k, head_dim, BW_R, sk, kv_heads, batch, k_ss, k_sh, k_sb);
  if (rc == TPB_OK) rc = fa_tmap(&v128, v, head_dim, BW_R, sk, kv_heads, batch, v_ss, v_sh, v_sb);
  if (rc == TPB_OK) rc = fa_tmap(&q64, q, head_dim, BW_T, sq, q_heads, batch, q_ss, q_sh, q_sb);
  if (rc == TPB_OK) rc = fa_tmap(&do64, dout, head_dim, BW_T, sq, q_heads, batch, do_ss, do_sh, do_sb);
  if (rc == TPB_OK) rc = fa_tmap(&k64, k, head_dim, BW_T, sk, kv_heads, batch, k_ss, k_sh, k_sb);
  if (rc == TPB_OK) rc = fa_tmap(&v64, v, head_dim, BW_T, sk, kv_heads, batch, v_ss, v_sh, v_sb);
  if (rc != TPB_OK) return rc;
  BwParams p;
  memset(&p, 0, sizeof(p));
  p.sq = sq; p.sk = sk; p.q_heads = q_heads; p.kv_heads = kv_heads; p.causal = causal;
  p.scale = scale;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.lse = lse;
  p.delta = delta;
  p.status = static_cast<uint32_t*>(status);
  p.bias = bias;
  p.bias_kind = !bias ? 0 : (bias_dtype == 1 ? 1 : 2);
  p.b_sb = bias_sb; p.b_sh = bias_sh; p.b_sq = bias_sq; p.b_sk = bias_sk;
  p.bias_vec = bias && bias_vector_rows(bias, bias_sb, bias_sh, bias_sq, bias_sk) && !(reinterpret_cast<uintptr_t>(dbias) & 15);
  p.dbias = nullptr;  // (the dK / dV launch leaves it alone)
  p.inv_scale = scale > 0.f ? 1.f / scale : 0.f;
  // dK / dV: the dk strides serve dv too (the existing contract)
  p.out0 = static_cast<bf16*>(dk); p.o0_sb = dk_sb; p.o0_ss = dk_ss; p.o0_sh = dk_sh;
  p.out1 = static_cast<bf16*>(dv); p.o1_sb = dk_sb; p.o1_ss = dk_ss; p.o1_sh = dk_sh;
  dim3 grid_kv((sk + BW_R - 1) / BW_R, kv_heads, batch);
  // a dense bf16 bias travels by TMA (strides and base are multiples of 16 bytes); fp32 ones, unaligned rows and masks that
  // broadcast over the queries are loaded element by element
  const int bias_mode = !bias ? 0 : (p.bias_kind == 2 && p.bias_vec && bias_sq > 0 && bias_sb >= 0 && bias_sh >= 0 ? 2 : 1);
  const bool kv_two = two_per_sm(head_dim, sk, kv_heads, batch, causal), q_two = two_per_sm(head_dim, sq, q_heads, batch, causal) || (bias_mode == 0 && dq_two_per_sm_128(head_dim, sq, sk, q_heads, batch));
  const int kv_rows = kv_two ? BW_T : step_rows(head_dim, bias_mode, sq, kv_heads, batch), q_rows = q_two ? BW_T : step_rows(head_dim, bias_mode, sk, q_heads, batch);
  CUtensorMap b_kv = q64, b_q = q64;
  if (bias_mode == 2) {  // (a wide dQ step takes two boxes)
    rc = fa_bias_tmap(&b_kv, bias, batch, q_heads, sq, sk, bias_sb, bias_sh, bias_sq, kv_rows, BW_R, false);
    if (rc == TPB_OK) rc = fa_bias_tmap(&b_q, bias, batch, q_heads, sq, sk, bias_sb, bias_sh, bias_sq, BW_R, BW_T, true);
    if (rc != TPB_OK) return rc;
  }
  auto launch = [&](auto dkv, const CUtensorMap& r1, const CUtensorMap& r2, const CUtensorMap* t1, const CUtensorMap* t2, const CUtensorMap& tb, dim3 grid) {
    constexpr bool DKV = decltype(dkv)::value;
    const bool wide = (DKV ? kv_rows : q_rows) == 128;
#define BW_ONE(D, BIAS)                                                                  \
  (wide ? bw_launch_wide<D, DKV, BIAS, 128>(r1, r2, t1[1], t2[1], tb, p, grid, s)        \
        : bw_launch<D, DKV, BIAS>(r1, r2, t1[0], t2[0], tb, p, grid, s))
    if (head_dim == 64 && (DKV ? kv_two : q_two)) {
#define BW_TWO(BIAS) bw_launch_wide<64, DKV, BIAS, 64>(r1, r2, t1[0], t2[0], tb, p, grid, s)
      return bias_mode == 0 ? BW_TWO(0) : bias_mode == 1 ? BW_TWO(1) : BW_TWO(2);
#undef BW_TWO
    }
    if (head_dim == 64) return bias_mode == 0 ? BW_ONE(64, 0) : bias_mode == 1 ? BW_ONE(64, 1) : BW_ONE(64, 2);
    if constexpr (!DKV) {
      if (bias_mode == 0 && q_two) return bw_launch_wide<128, DKV, 0, 64>(r1, r2, t1[0], t2[0], tb, p, grid, s);
    }
    return bias_mode == 0   ? BW_ONE(128, 0)
           : bias_mode == 1 ? bw_launch<128, DKV, 1>(r1, r2, t1[0], t2[0], tb, p, grid, s)
                            : bw_launch<128, DKV, 2>(r1, r2, t1[0], t2[0], tb, p, grid, s);
#undef BW_ONE
  };
  const CUtensorMap qs[2] = {q64, q128}, dos[2] = {do64, do128}, ks[2] = {k64, k128}, vs[2] = {v64, v128};  // steps of 64 and of 128 rows
  rc = launch(std::true_type{}, k128, v128, qs, dos, b_kv, grid_kv);
  if (rc != TPB_OK) return rc;
  p.out0 = static_cast<bf16*>(dq); p.o0_sb = dq_sb; p.o0_ss = dq_ss; p.o0_sh = dq_sh;
  p.out1 = nullptr;
  p.dbias = dbias;
  return launch(std::false_type{}, q128, do128, ks, vs, b_q, dim3((sq + BW_R - 1) / BW_R, q_heads, batch));
}

// Gradient of a bf16 score bias that the batches share (bias_sb = 0; bias_sh = 0: the heads as well), for head_dim 64: dbias has the bias' strides and
// is written, not added to.  lse, delta: [batch][q_heads][sq], delta as tpb_attn_backward_sm100 left it.  Other arguments as there.
extern "C" int tpb_attn_bias_grad_sm100(const void* q, const void* k, const void* v, const void* dout, const float* lse, const float* delta, int batch, int sq,
                                        int sk, int q_heads, int kv_heads, int head_dim, long long q_sb, long long q_ss, long long q_sh, long long k_sb,
                                        long long k_ss, long long k_sh, long long v_sb, long long v_ss, long long v_sh, long long do_sb, long long do_ss,
                                        long long do_sh, int causal, float scale, const void* bias, long long bias_sh, long long bias_sq, void* dbias,
                                        int dbias_fp32, void* status, void* stream_) {
  if (!q || !k || !v || !dout || !lse || !delta || !bias || !dbias || !status || batch <= 0 || sq <= 0 || sk <= 0 || q_heads <= 0 || kv_heads <= 0 ||
      q_heads % kv_heads || bias_sq <= 0 || bias_sh < 0 || !(scale > 0.f))
    return TPB_ERR_ARG;
  const int q_tiles = (sq + BW_R - 1) / BW_R, k_tiles = (sk + BG_KEYS - 1) / BG_KEYS, planes = bias_sh ? q_heads : 1;
  if (head_dim != 64 || q_tiles > 65535 || planes > 65535) return TPB_ERR_SIZE;
  const long long strides[] = {q_ss, k_ss, v_ss, do_ss, q_heads > 1 ? q_sh : 0, q_heads > 1 ? do_sh : 0, kv_heads > 1 ? k_sh : 0,
                               kv_heads > 1 ? v_sh : 0, batch > 1 ? q_sb : 0, batch > 1 ? k_sb : 0, batch > 1 ? v_sb : 0, batch > 1 ? do_sb : 0, bias_sh, bias_sq};
  for (long long s : strides)
    if (s & 7) return TPB_ERR_ALIGN;
  if (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)dout | (uintptr_t)bias | (uintptr_t)dbias) & 15) return TPB_ERR_ALIGN;
  if (fa_bind_thread() != TPB_OK) return TPB_ERR_CUDA;
  CUtensorMap tq, tdo, tk, tv;
  int rc = fa_tmap(&tq, q, head_dim, BW_R, sq, q_heads, batch, q_ss, q_sh, q_sb);
  if (rc == TPB_OK) rc = fa_tmap(&tdo, dout, head_dim, BW_R, sq, q_heads, batch, do_ss, do_sh, do_sb);
  if (rc == TPB_OK) rc = fa_tmap(&tk, k, head_dim, BG_KEYS, sk, kv_heads, batch, k_ss, k_sh, k_sb);
  if (rc == TPB_OK) rc = fa_tmap(&tv, v, head_dim, BG_KEYS, sk, kv_heads, batch, v_ss, v_sh, v_sb);
  if (rc != TPB_OK) return rc;
  BgParams p;
  memset(&p, 0, sizeof(p));
  p.batch = batch; p.sq = sq; p.sk = sk; p.q_heads = q_heads; p.kv_heads = kv_heads; p.causal = causal;
  p.scale_log2e = scale * 1.4426950408889634f;
  p.lse = lse;
  p.delta = delta;
  p.bias = static_cast<const bf16*>(bias);
  p.dbias = dbias;
  p.dbias_fp32 = dbias_fp32;
  p.b_sh = bias_sh; p.b_sq = bias_sq;
  p.status = static_cast<uint32_t*>(status);
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TPB_ERR_CUDA;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(attn_bias_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(BG_SMEM)) != cudaSuccess) return TPB_ERR_CUDA;
    configured[dev].store(true, std::memory_order_release);
  }
  attn_bias_grad_kernel<<<dim3(k_tiles, q_tiles, planes), BG_THREADS, BG_SMEM, static_cast<cudaStream_t>(stream_)>>>(tq, tdo, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? TPB_OK : TPB_ERR_CUDA;
}
