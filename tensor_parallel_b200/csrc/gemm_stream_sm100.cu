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
// A decode step of four 7B layers and the head (batch 8, 2048-token context) went from 793 to 575 us with this kernel and the
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

constexpr int GS_UNIT = StreamRows::UNIT;
constexpr int GS_BK = 64;        // columns of a box: 128-byte swizzled rows
constexpr int GS_THREADS = 192;
constexpr int GS_EPI = 128;
constexpr int GS_MAX_STAGES = 16;
__host__ __device__ constexpr size_t GS_SLICE_BYTES(int ks) { return ks > 1 ? 9 * 1024 : 0; }

struct GsParams {
  int features, tokens, k_stages;
  StreamRows rows;      // (a stage's layout follows its pass_units; tmap_w loads boxes of its box_units, tmap_w1 of one unit)
  int slice_cols;       // KS > 1: columns of a slice
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
// KBOX boxes of 64 columns per stage and unit.
// KS > 1 (every CTA has one unit): the 32 rows alone would leave three quarters of an MMA's rows to garbage, and a long chain of
// such MMAs, about 55 clocks each, is slower than the weights arrive (4096 x 11008: 688 of them, 20 us; the weights need 14).
// So the contraction is cut into KS slices that run side by side: weight slice s fills rows 32 s .. of the tile, token slice s
// columns TOK s .., the diagonal blocks of the product are the slices' partial sums (the other blocks are never read), and
// the epilogue adds them up through shared memory.
template <int BN, int NACC, int KBOX, int KS>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_stream_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_w1, const __grid_constant__ CUtensorMap tmap_x,
                   const GsParams p) {
  constexpr uint32_t X_BOX = BN * GS_BK * 2, X_BYTES = KBOX * X_BOX;
  constexpr uint32_t ACC_COLS = NACC * BN, TMEM_COLS = 2 * ACC_COLS;  // two accumulator sets: a pass's epilogue runs under the next
  constexpr int STEPS = KBOX * (GS_BK / 16);  // MMAs of a stage; step n of the pass goes to accumulator n % NACC
  static_assert(TMEM_COLS <= 512 && (TMEM_COLS & (TMEM_COLS - 1)) == 0 && TMEM_COLS >= 32, "TMEM allocation");
  constexpr int TOK = BN / KS;  // token columns of a slice
  const uint32_t w_box = uint32_t(KS > 1 ? KS : p.rows.pass_units) * GS_UNIT * 128;  // [rows of a pass, or of all slices][64 columns]
  const uint32_t w_bytes = KBOX * w_box, stage_bytes = w_bytes + X_BYTES;

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
  float* slices = reinterpret_cast<float*>(smem + 1024);        // KS > 1: [KS][32 rows][TOK + 1] partial sums
  uint8_t* ring = smem + 1024 + GS_SLICE_BYTES(KS);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // (known to be uniform)
  const int unit0 = p.rows.first(blockIdx.x), my_units = p.rows.first(blockIdx.x + 1) - unit0, passes = p.rows.passes;
  auto pass_start = [&](int i) { return p.rows.pass_start(unit0, my_units, i); };
  auto pass_units = [&](int i) { return pass_start(i + 1) - pass_start(i); };

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_w);
    prefetch_tmap(&tmap_w1);
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
    // ---------------- TMA producer (the warp stays together, one lane issues) ----------------
    const uint32_t leader = elect_one();
    struct Stage { int pass, ks, s; uint32_t parity; };
    auto advance = [&](Stage& i) {
      if (++i.ks == p.k_stages) { i.ks = 0; ++i.pass; }
      if (++i.s == p.stages) { i.s = 0; i.parity ^= 1; }
    };
    auto load_w = [&](const Stage& i) {
      const int u = pass_units(i.pass), row0 = pass_start(i.pass) * GS_UNIT, col0 = i.ks * KBOX * GS_BK;
      const uint32_t dst = smem_u32(ring + size_t(i.s) * stage_bytes);
      uint64_t* bar = &full_bar[i.s];
      mbar_expect_tx_lead(leader, bar, KBOX * uint32_t(KS > 1 ? KS : u) * GS_UNIT * 128 + X_BYTES);
      if (KS > 1) {
#pragma unroll
        for (int j = 0; j < KBOX; ++j)
#pragma unroll
          for (int sl = 0; sl < KS; ++sl)
            tma_load_2d_lead(leader, dst + j * w_box + sl * GS_UNIT * 128, &tmap_w1, bar, sl * p.slice_cols + col0 + j * GS_BK, row0);
        return;
      }
      int done = 0;
      for (; done + p.rows.box_units <= u; done += p.rows.box_units) {
#pragma unroll
        for (int j = 0; j < KBOX; ++j)  // (columns and rows past the end arrive as zeros)
          tma_load_2d_lead(leader, dst + j * w_box + done * GS_UNIT * 128, &tmap_w, bar, col0 + j * GS_BK, row0 + done * GS_UNIT);
      }
      for (; done < u; ++done) {
#pragma unroll
        for (int j = 0; j < KBOX; ++j)
          tma_load_2d_lead(leader, dst + j * w_box + done * GS_UNIT * 128, &tmap_w1, bar, col0 + j * GS_BK, row0 + done * GS_UNIT);
      }
    };
    auto load_x = [&](const Stage& i) {
      const uint32_t dst = smem_u32(ring + size_t(i.s) * stage_bytes + w_bytes);
#pragma unroll
      for (int j = 0; j < KBOX; ++j)
#pragma unroll
        for (int sl = 0; sl < KS; ++sl)
          tma_load_2d_lead(leader, dst + j * X_BOX + sl * TOK * 128, &tmap_x, &full_bar[i.s], sl * p.slice_cols + (i.ks * KBOX + j) * GS_BK, 0);
    };
    const int total = passes * p.k_stages, ahead = min(total, p.stages);
    Stage w = {0, 0, 0, 0}, x = w;  // (parity: round of the ring, a stage is free again after the round before)
    for (int n = 0; n < ahead; ++n, advance(w)) load_w(w);
    pdl_wait();
    pdl_trigger();
    for (int n = 0; n < ahead; ++n, advance(x)) load_x(x);
    for (int n = ahead; n < total; ++n, advance(w)) {
      const bool free_stage = !*abort_flag && mbar_wait(&empty_bar[w.s], w.parity ^ 1);
      if (!__all_sync(0xffffffffu, free_stage)) {
        if (leader) give_up();
        break;
      }
      load_w(w);
      load_x(w);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the warp stays together, one lane issues: see umma_bf16_lead) ----------------
    const uint32_t leader = elect_one();
    int s = 0;
    uint32_t parity = 0;
    for (int pass = 0; pass < passes; ++pass) {
      const int acc = pass & 1;
      const bool free_acc = !*abort_flag && mbar_wait(&acc_empty[acc], ((pass >> 1) & 1) ^ 1);
      if (!__all_sync(0xffffffffu, free_acc)) {
        if (leader) give_up();
        break;
      }
      tc_fence_after();
      const int u = pass_units(pass);
      const uint32_t idesc = make_idesc_bf16((KS == 1 && u * GS_UNIT <= 64 && p.act != 5) ? 64 : 128, BN);
      const uint32_t d_tmem = tmem_base + acc * ACC_COLS;
      bool ok = true;
      for (int ks = 0; ks < p.k_stages; ++ks) {
        const bool full = mbar_wait(&full_bar[s], parity);
        if (!__all_sync(0xffffffffu, full)) {
          if (leader) give_up();
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t w_addr = smem_u32(ring + size_t(s) * stage_bytes);
        const uint32_t w_lo = desc_kmajor_lo(w_addr), x_lo = desc_kmajor_lo(w_addr + w_bytes);
#pragma unroll
        for (int j = 0; j < KBOX; ++j) {
#pragma unroll
          for (int kk = 0; kk < GS_BK / 16; ++kk) {
            const int n = j * (GS_BK / 16) + kk;
            const uint32_t d = STEPS % NACC == 0 ? (n % NACC) * BN : ((ks * STEPS + n) % NACC) * BN;
            umma_bf16_lead(leader, d_tmem + d, w_lo + j * (w_box >> 4) + kk * 2, x_lo + j * (X_BOX >> 4) + kk * 2, idesc,
                           ks * STEPS + n >= NACC ? 1u : 0u);
          }
        }
        umma_commit_lead(leader, &empty_bar[s]);
        if (++s == p.stages) { s = 0; parity ^= 1; }
      }
      if (!ok) break;
      umma_commit_lead(leader, &acc_full[acc]);
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
    const bool pitch_even = (p.ld_out & 1) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 3) == 0;
    // Finishes the value x of (token t, feature m) and stores it; called by a whole warp, neighbouring lanes own neighbouring features.
    auto finish = [&](float x, int t, int m, bool m_ok, float bias, float rowsum, float res) {
      if (p.norm_mode) x = x * norm_stats[2 * t] - norm_stats[2 * t + 1] * rowsum;
      x += bias;
      if (gated) {
        // lanes 0-15 of a warp hold gate rows, lanes 16-31 the matching up rows
        const float partner = __shfl_xor_sync(0xffffffffu, x, 16);
        const size_t idx = size_t(t) * p.ld_out + (m >> 5) * 16 + (m & 15);
        if (m_ok && lane < 16 && TPB_IN_BOUNDS(idx < p.out_elems, p.status)) p.out[idx] = __float2bfloat16(x / (1.f + __expf(-x)) * partner);
        return;
      }
      if (p.act) x = gs_act(x, p.act);
      x += res;
      // pairs of neighbouring lanes store two features (4 bytes) at a time
      const bool writes_pair = pitch_even && !(lane & 1) && m + 1 < p.features;
      const bool covered = pitch_even && (lane & 1);  // the even neighbour stores this lane's value
      const float up = __shfl_down_sync(0xffffffffu, x, 1);
      const size_t idx = size_t(t) * p.ld_out + m;
      if (m_ok && TPB_IN_BOUNDS(idx + (writes_pair ? 1 : 0) < p.out_elems, p.status)) {
        if (writes_pair) *reinterpret_cast<uint32_t*>(p.out + idx) = pack_bf16x2(x, up);
        else if (!covered) p.out[idx] = __float2bfloat16(x);
      }
    };
    const int n_acc = min(NACC, p.k_stages * STEPS);
    if constexpr (KS > 1) {
      constexpr int MINE = TOK / KS;  // tokens this warp finishes: the slices' sums are exchanged, then each warp takes a share
      const int m = unit0 * GS_UNIT + lane;
      const bool m_ok = m < p.features;
      const float bias = (p.bias && m_ok) ? p.bias_scale * __bfloat162float(p.bias[m]) : 0.f;
      const float rowsum = (p.norm_rowsum && m_ok) ? p.norm_rowsum[m] : 0.f;
      float res[MINE];
#pragma unroll
      for (int j = 0; j < MINE; ++j) {
        const int t = quarter * MINE + j;
        res[j] = (p.residual && m_ok && t < p.tokens) ? __bfloat162float(p.residual[size_t(t) * p.ld_out + m]) : 0.f;
      }
      const bool ready = !*abort_flag && mbar_wait(&acc_full[0], 0);
      if (!ready) give_up();
      tc_fence_after();
      if (__all_sync(0xffffffffu, ready)) {
        // this warp's TMEM lanes are the 32 rows of slice `quarter`; its columns of the product are [TOK quarter, TOK quarter + TOK)
        float v[TOK];
#pragma unroll
        for (int j = 0; j < TOK; ++j) v[j] = 0.f;
        for (int a = 0; a < n_acc; ++a) {
          uint32_t r[16];  // (TOK = 8: the upper half belongs to the next slice, or to the next accumulator; it is not used)
          tmem_ld_x16(tmem_base + (uint32_t(quarter * 32) << 16) + a * BN + quarter * TOK, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < TOK; ++j) v[j] += __uint_as_float(r[j]);
        }
#pragma unroll
        for (int j = 0; j < TOK; ++j) slices[(quarter * 32 + lane) * (TOK + 1) + j] = v[j];
      }
      asm volatile("bar.sync 1, %0;" ::"n"(GS_EPI) : "memory");
      if (!*abort_flag) {
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
          const int t = quarter * MINE + j;
          if (t >= p.tokens) break;  // (uniform)
          float x = 0.f;
#pragma unroll
          for (int sl = 0; sl < KS; ++sl) x += slices[(sl * 32 + lane) * (TOK + 1) + t];
          finish(x, t, m, m_ok, bias, rowsum, res[j]);
        }
      }
    } else {
    for (int pass = 0; pass < passes; ++pass) {
      const int acc = pass & 1, rows = pass_units(pass) * GS_UNIT;
      const bool m64 = rows <= 64 && !gated;
      // TMEM lane -> row of the pass: lane for M = 128; with M = 64 the first 16 lanes of each quarter hold 16 rows
      const int local_row = m64 ? quarter * 16 + lane : quarter * 32 + lane;
      const int m = pass_start(pass) * GS_UNIT + local_row;
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
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (n0 + j >= p.tokens) break;  // (uniform)
          finish(v[j], n0 + j, m, m_ok, bias, rowsum, res[j]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[acc]);
    }
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Ring of a CTA.  As deep as one CTA per SM allows: with 112 KB two consecutive kernels can share an SM, but a decode step of four
// 7B layers then takes 618 us, with 144 / 170 / 204 KB 591 / 582 / 575 us.
constexpr size_t GS_RING_BYTES = 204 * 1024;

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

template <int BN, int NACC, int KBOX, int KS>
static int gs_launch(const StreamGemm& g, int sms, cudaStream_t stream) {
  GsParams p;
  memset(&p, 0, sizeof(p));
  p.features = g.features;
  p.tokens = g.tokens;
  p.k_stages = ((g.k + KS - 1) / KS + KBOX * GS_BK - 1) / (KBOX * GS_BK);  // (of a slice)
  p.slice_cols = p.k_stages * KBOX * GS_BK;
  p.rows = gemm_stream_rows(g.features, sms);
  const size_t w_box = size_t(KS > 1 ? KS : p.rows.pass_units) * GS_UNIT * 128;
  const size_t stage_bytes = size_t(KBOX) * (w_box + BN * GS_BK * 2);
  // an MMA of M = 64 / 128 rows reads that many rows from the last weight box of the ring: what lies behind the last token box
  const size_t need = size_t(128) * 128, have = w_box + size_t(KBOX) * BN * GS_BK * 2;
  const size_t over = need > have ? need - have : 0;
  int stages = int(GS_RING_BYTES / stage_bytes);
  if (stages > GS_MAX_STAGES) stages = GS_MAX_STAGES;
  if (stages < 2) stages = 2;
  p.stages = stages;
  const size_t smem = 1024 + 1024 + GS_SLICE_BYTES(KS) + stages * stage_bytes + over;
  static std::atomic<bool> configured[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return TPB_ERR_CUDA;
  if (!configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(gemm_stream_kernel<BN, NACC, KBOX, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return TPB_ERR_CUDA;
    configured[dev].store(true, std::memory_order_release);
  }
  CUtensorMap tw, tw1, tx;
  int rc = gs_tmap(&tw, g.w, g.features, g.k, g.ldw, p.rows.box_units * GS_UNIT);
  if (rc == TPB_OK) rc = gs_tmap(&tw1, g.w, g.features, g.k, g.ldw, GS_UNIT);
  if (rc == TPB_OK) rc = gs_tmap(&tx, g.x, g.tokens, g.k, g.ldx, BN / KS);
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
  return launch_dependent(gemm_stream_kernel<BN, NACC, KBOX, KS>, dim3(p.rows.grid), dim3(GS_THREADS), smem, stream, g.early != 0 || pdl_enabled(), tw, tw1, tx, p) ==
                 cudaSuccess
             ? TPB_OK
             : TPB_ERR_CUDA;
}

bool gemm_stream_fits(int features, int k, int sms) {
  const long long unit_bytes = 2LL * GS_UNIT * k;
  return (features + GS_UNIT - 1) / GS_UNIT >= sms / 2 || unit_bytes <= 1024 * 1024;
}

// 512 contiguous bytes of every weight row per stage where rows are long and a stage stays small, else 256 in twice as many stages:
// 8192 x 40960 (two units per CTA) 101 us with 512 bytes and 117 us with 256, 32768 x 8192 (seven) 85 and 83 us, a decode step of
// four 7B layers (rows of 8 KB) 587 and 575 us.
template <int BN, int NACC>
static int gs_pick(const StreamGemm& g, int sms, cudaStream_t stream) {
  const bool small = (g.features + GS_UNIT - 1) / GS_UNIT <= 2 * sms;
  return g.k >= 8192 && small ? gs_launch<BN, NACC, 4, 1>(g, sms, stream) : gs_launch<BN, NACC, 2, 1>(g, sms, stream);
}

int gemm_stream_launch(const StreamGemm& g, int sms, cudaStream_t stream) {
  // one unit per CTA: slices of the contraction side by side, as long as each has a few stages (4096 x 4096 11.8 -> 7.9 us, 4096 x 11008
  // 22.1 -> 16.6 us, 1536 x 4096 10.2 -> 6.0 us; more than 16 tokens would need more than 64 MMA columns)
  const bool one_unit = (g.features + GS_UNIT - 1) / GS_UNIT <= sms && g.k >= 1024;
  if (one_unit && g.tokens <= 8) return gs_launch<32, 4, 2, 4>(g, sms, stream);
  if (one_unit && g.tokens <= 16) return gs_launch<64, 2, 2, 4>(g, sms, stream);
  if (g.tokens <= 16) return gs_pick<16, 8>(g, sms, stream);
  if (g.tokens <= 32) return gs_pick<32, 8>(g, sms, stream);
  if (g.tokens <= 64) return gs_pick<64, 2>(g, sms, stream);
  return TPB_ERR_ARG;
}

cudaError_t gemm_stream_preload() {
  cudaFuncAttributes attr;
  cudaError_t e = cudaSuccess;
#define LOAD(BN, NACC, KBOX, KS) if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, gemm_stream_kernel<BN, NACC, KBOX, KS>)
  LOAD(16, 8, 2, 1); LOAD(32, 8, 2, 1); LOAD(64, 2, 2, 1); LOAD(16, 8, 4, 1); LOAD(32, 8, 4, 1); LOAD(64, 2, 4, 1);
  LOAD(32, 4, 2, 4); LOAD(64, 2, 2, 4);
#undef LOAD
  return e;
}

}  // namespace tpb

// The decomposition of a few-token GEMM, for tests: shape = {units, grid, passes, pass_units, box_units}, and at starts[0 .. passes] the
// units at which the passes of CTA `cta` begin and the last one ends (room for `capacity` of them).
extern "C" int tpb_gemm_stream_rows(int features, int sms, int cta, int* shape, int* starts, int capacity) {
  if (features <= 0 || sms <= 0 || cta < 0 || !shape || !starts) return TPB_ERR_ARG;
  const tpb::StreamRows r = tpb::gemm_stream_rows(features, sms);
  if (cta >= r.grid || r.passes >= capacity) return TPB_ERR_ARG;
  const int values[5] = {r.units, r.grid, r.passes, r.pass_units, r.box_units};
  memcpy(shape, values, sizeof(values));
  const int unit0 = r.first(cta), mine = r.first(cta + 1) - unit0;
  for (int i = 0; i <= r.passes; ++i) starts[i] = r.pass_start(unit0, mine, i);
  return TPB_OK;
}
