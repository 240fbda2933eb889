// Interface between the GEMM planner / entry points (gemm_sm100.cu) and the CTA-pair kernel (gemm_pair_sm100.cu).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace tpb {

struct PairGemm {
  const void* x;   // tokens operand: [tokens, k] (pitch ldx), or [k, tokens] when x_mn
  const void* w;   // weights operand: [features, k] (pitch ldw), or [k, features] when w_mn
  int tokens, features, k, ldx, ldw;
  int x_mn, w_mn;
  __nv_bfloat16* out;
  int ld_out;
  const __nv_bfloat16* bias;
  float bias_scale;
  const __nv_bfloat16* residual;
  int act;
  uint32_t* status;
  size_t out_elems;
};

// Columns of the pair tile (256 or 128) a many-token GEMM of this shape should use, or 0 when single-CTA tiles are faster.
int gemm_pair_tile(int tokens, int features, int sms);
int gemm_pair_launch(const PairGemm& g, int bn, int sms, cudaStream_t stream);
cudaError_t gemm_pair_preload();

}  // namespace tpb
