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

// True if a few-token (at most 64) GEMM of this shape streams its weights on one pass of row ranges, false if split-K tiles
// are the better decomposition.
bool gemm_stream_fits(int features, int k, int sms);
int gemm_stream_launch(const StreamGemm& g, int sms, cudaStream_t stream);
cudaError_t gemm_stream_preload();

}  // namespace tpb
