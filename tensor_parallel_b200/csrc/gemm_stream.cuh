// Interface between the GEMM planner / entry points (gemm_sm100.cu) and the few-token kernel (gemm_stream_sm100.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace tpb {

struct StreamGemm {
  const void* x;   // [tokens, k], pitch ldx
  const void* w;   // [features, k], pitch ldw
  int tokens, features, k, ldx, ldw;
  __nv_bfloat16* out;
  int ld_out;
  const __nv_bfloat16* bias;
  float bias_scale;
  const __nv_bfloat16* residual;
  int act;
  int norm_mode;   // 0 none, 1 RMSNorm, 2 LayerNorm of the token rows (see tpb_gemm_opts_t)
  float norm_eps;
  const __nv_bfloat16* norm_x;
  long long norm_ld;
  int norm_k;
  const float* norm_rowsum;
  int early;       // launch as a programmatic dependent and fetch weights before the previous kernel has finished
  uint32_t* status;
  size_t out_elems;
};

// How the rows of the weight are dealt out, in units of 32: CTA c of `grid` owns the units [first(c), first(c + 1)) and walks them in
// `passes` passes, the same number everywhere and of even length (a short pass behind a full one would stream with most of the ring
// empty: 22016 rows, 4 or 5 units per CTA, 4 + 1 units 39 us, 2 + 3 units 33 us).
struct StreamRows {
  static constexpr int UNIT = 32;      // rows of a unit; the gated activation pairs 16 gate rows with their 16 up rows
  static constexpr int PASS_UNITS = 4;  // 128 rows: the lanes of TMEM
  int units, grid, passes;
  int pass_units;  // units of the longest pass of any CTA
  int box_units;   // of the shortest: every pass is at least one box of this many units
  __host__ __device__ int first(int cta) const { return int((long long)cta * units / grid); }
  // unit at which pass i of a CTA that owns `mine` units from `unit0` on starts (i == passes: where the last one ends)
  __host__ __device__ int pass_start(int unit0, int mine, int i) const { return unit0 + mine * i / passes; }
};
inline StreamRows gemm_stream_rows(int features, int sms) {
  StreamRows r;
  r.units = (features + StreamRows::UNIT - 1) / StreamRows::UNIT;
  r.grid = r.units < sms ? r.units : sms;
  const int most = (r.units + r.grid - 1) / r.grid, least = r.units / r.grid;  // units of the longest and the shortest range
  r.passes = (most + StreamRows::PASS_UNITS - 1) / StreamRows::PASS_UNITS;
  r.pass_units = (most + r.passes - 1) / r.passes;
  r.box_units = least / r.passes;
  return r;
}

// True if a few-token (at most 64) GEMM of this shape streams its weights on one pass of row ranges, false if split-K tiles
// are the better decomposition.
bool gemm_stream_fits(int features, int k, int sms);
int gemm_stream_launch(const StreamGemm& g, int sms, cudaStream_t stream);
cudaError_t gemm_stream_preload();

}  // namespace tpb
