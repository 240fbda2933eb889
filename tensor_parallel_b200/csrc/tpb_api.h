// C ABI of libtpb200: every entry point is extern "C", takes raw device pointers plus a CUDA stream
// handle, launches asynchronously on that stream and returns one of the TPB_* codes below.
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

enum {
  TPB_OK = 0,
  TPB_ERR_ARG = 1,        // null pointer / non-positive size / unsupported value
  TPB_ERR_ALIGN = 2,      // pointer or leading dimension violates an alignment rule (TMA needs 16 bytes)
  TPB_ERR_CUDA = 3,       // a CUDA runtime call failed (see cudaGetLastError)
  TPB_ERR_DRIVER = 4,     // a driver entry point is unavailable
  TPB_ERR_TMAP = 5,       // cuTensorMapEncodeTiled rejected the descriptor
  TPB_ERR_WORKSPACE = 6,  // reduction workspace too small for this shape
  TPB_ERR_SIZE = 7,       // size beyond a compiled-in maximum
};

#define TPB_MAX_WORLD 8
#define TPB_COMM_MAX_BLOCKS 160  // largest grid of a stand-alone collective = rows of its signal arrays (one CTA per SM and more)
#define TPB_COMM_LL_MAX_WORDS 32768  // 16-byte words (8 payload bytes each) per rank and parity in the flagged-word area

typedef struct {
  int swapped;  // 1: weight rows fill the 128 tensor-core rows (few tokens), 0: tokens do
  int bn;       // accumulator columns per tile
  int kbox;     // 64-column k-blocks fetched per pipeline stage (k_blocks / kb_per_split count stages)
  int m_tiles, n_tiles, k_blocks, k_splits, kb_per_split;
  int reduce;   // partial tiles go through the slot workspace (split-K and / or several ranks)
  int grid;
  int tokens_pad;
  int tiles;
  size_t slot_elems;  // fp32 elements one slot must hold
  int stream_k;       // 1: the (tile, k-block) units are dealt out as one contiguous range per CTA; k_splits then is an
                      // upper bound of the CTAs that contribute to one tile
  int pair;           // columns of the CTA-pair tile (256 or 128) when the many-token pair kernel runs this shape, else 0
  int stream;         // 1: the few-token weight-streaming kernel runs this shape (the tile fields then describe its fallback)
} tpb_gemm_plan_t;

// Workspace of the fused split-K / all-reduce epilogue.  All pointers are device pointers valid on the
// launching GPU; slots[d] / arrivals[d] point into rank d's memory (peer-mapped for d != rank).
typedef struct {
  int world, rank;
  void* slots[TPB_MAX_WORLD];     // fp32 [max_slots][slot_stride]; needs world + k_splits slots
  void* arrivals[TPB_MAX_WORLD];  // uint32 [max_tiles]
  void* expected;                 // local uint32 [max_tiles]
  void* split_counters;           // local uint32 [max_tiles], zero-initialised
  void* status;                   // local uint32 status word
  size_t slot_stride;             // elements per slot
  int max_slots, max_tiles;
  void* ll_epochs;                // local uint32 [max_tiles], zero-initialised: epochs of the flagged-word exchange that small
                                  // cross-rank sums use (needs max_slots >= 32 + 2 * world); null selects arrival counters
  void* mc_slots;                 // NVLink multicast alias of slots[*] (the same offsets reach every rank's workspace): the flagged
                                  // words are then pushed with one multimem.st instead of one store per rank; null: peer stores
} tpb_reduce_ctx_t;

// Operands of the fused all-gather + GEMM (see tpb_gemm_allgather_bf16).
typedef struct {
  int world, rank;
  const void* local;                  // this rank's column slice [tokens, cols_local] bf16
  int local_ld, cols_local;
  void* gathered[TPB_MAX_WORLD];      // every rank's gathered buffer [tokens, world * cols_local] (peer-mapped)
  void* flags[TPB_MAX_WORLD];         // every rank's arrival words, uint32 [world], indexed by source rank
  void* push_counter;                 // local uint32, zero-initialised
  unsigned epoch;                     // number of fused all-gather calls issued on these flags, this one included
  void* mc_gathered;                  // multicast (NVLS) view of the gathered buffers, or null: the slice is then pushed with
                                      // one plain store per peer instead of one multimem.st
} tpb_allgather_ctx_t;

// Options of tpb_gemm_bf16_ex.
typedef struct {
  int x_mn, w_mn;            // the operand lies transposed in memory: x as [k, tokens] (row pitch ldx), w as [k, features]
                             // (row pitch ldw).  Needs a plan made with flag bit 0 (tokens on the tensor-core rows).
  int norm_mode;             // 0 none, 1 RMSNorm, 2 LayerNorm of the rows of x, folded into the kernel (<= 64 tokens):
                             // x must be the UNNORMALISED rows, w must already carry the norm weight (w'[f, k] = w[f, k] g[k])
                             // and the result is rstd (x w'^T - mean rowsum) + bias_scale * bias
  float norm_eps;
  const void* norm_x;        // rows the statistics are taken over: x itself, or (norm_k > k) the full rows x is a column
                             // slice of (a row-parallel projection of a normalised state)
  long long norm_ld;
  int norm_k;                // columns of norm_x; <= 0: k
  const float* norm_rowsum;  // LayerNorm: fp32 [features], sum over k of w'[f, k]; the caller folds W beta into the bias
  double wait_seconds;       // bound of the waits for peer GPUs; <= 0: the library default (tpb_set_wait_limit)
  size_t out_elems;          // extent of `out` in elements, for the index checks of a -DTPB_BOUNDS build; 0: derived from the shape
  int early;                 // launch as a programmatic dependent of the previous kernel of the stream and read w before that
                             // kernel has finished (few-token streaming kernel only): w must not be an output of that kernel
} tpb_gemm_opts_t;

// 1 if this library was built with -DTPB_BOUNDS (kernels check their store indices and report STATUS_BAD_ARG = 3 in the
// status word instead of touching memory outside the extents they were given).
int tpb_bounds_checked(void);

int tpb_gemm_plan(int tokens, int features, int k, int world, int force_splits, int force_kbox,
                  tpb_gemm_plan_t* plan);
int tpb_gemm_plan_ex(int tokens, int features, int k, int world, int force_splits, int force_kbox, int flags,
                     tpb_gemm_plan_t* plan);
int tpb_gemm_tune_split(int min_tile_kb, int target_kb);
int tpb_set_wait_limit(double seconds);

// out[tokens, features] = act(x[tokens, k] @ w[features, k]^T + bias_scale * bias) + residual
// (bf16 operands, fp32 accumulation).  With rc->world > 1 the product is additionally summed over all ranks
// inside the same kernel (every rank must launch it with the same shapes).  `residual` may be `out`: every element is read by the thread that
// then stores it, once its sum is complete.
int tpb_gemm_bf16(const void* x, const void* w, void* out, const void* bias, const void* residual, int tokens,
                  int features, int k, int ldx, int ldw, int ld_out, int act, float bias_scale,
                  const tpb_gemm_plan_t* plan, const tpb_reduce_ctx_t* rc, void* stream);

int tpb_gemm_bf16_ex(const void* x, const void* w, void* out, const void* bias, const void* residual, int tokens,
                     int features, int k, int ldx, int ldw, int ld_out, int act, float bias_scale,
                     const tpb_gemm_plan_t* plan, const tpb_reduce_ctx_t* rc, const tpb_gemm_opts_t* opts, void* stream);

int tpb_gemm_allgather_bf16(const void* w, void* out, const void* bias, int tokens, int features, int k, int ld_gathered,
                            int ldw, int ld_out, int act, const tpb_gemm_plan_t* plan, const tpb_reduce_ctx_t* rc,
                            const tpb_allgather_ctx_t* ag, void* stream);

// RMSNorm (mode 0) / LayerNorm (mode 1) of [rows, cols] bf16 (dtype 0) or fp32 (dtype 1) rows; cols a multiple of 8.  With `residual`,
// x + residual is normalised and also written to sum_out.  rstd_out / mean_out (fp32 per row) may be null.
int tpb_norm_fwd(const void* x, const void* residual, const void* weight, const void* bias, void* out, void* sum_out, float* rstd_out,
                 float* mean_out, int rows, int cols, float eps, int mode, int dtype, void* stream);
// Rows of fp32 partials [rows][cols] that part_w / part_b of tpb_norm_bwd hold.
int tpb_norm_bwd_parts(int rows, int cols);
// dweight / dbias (either may be null, with its partials) are written, not accumulated; grad_dtype: 0 = bf16, 1 = fp32.
int tpb_norm_bwd(const void* dy, const void* x, const void* weight, const float* rstd, const float* mean, void* dx, float* part_w,
                 float* part_b, void* dweight, void* dbias, int rows, int cols, int mode, int dtype, int grad_dtype, void* stream);

// Column sums in fp32 of g[rows, cols] (bf16, contiguous, 16-byte aligned, cols a multiple of 8), stored as bf16 (out_dtype 0) or fp32 (1); partials:
// fp32 [tpb_col_sum_parts(rows, cols)][cols], not needed for one part.
int tpb_col_sum_parts(int rows, int cols);
int tpb_col_sum(const void* g, void* out, float* partials, int rows, int cols, int out_dtype, void* stream);

// Sizes of the structures above as this library was built, one byte-count per 16 bits (plan, reduction context, options), for callers that
// are built apart from it.
#define TPB_API_LAYOUT ((unsigned long long)sizeof(tpb_gemm_plan_t) | (unsigned long long)sizeof(tpb_reduce_ctx_t) << 16 | (unsigned long long)sizeof(tpb_gemm_opts_t) << 32)
unsigned long long tpb_api_layout(void);

// Measurement aids.  tpb_gemm_debug caps the smem ring depth (0 restores the default).  Skipping the MMAs and the
// kernel-internal %globaltimer trace (tpb_gemm_trace / tpb_gemm_trace_read) exist only in a library built with
// -DTPB_GEMM_TRACE; in the product build they return TPB_ERR_ARG and the kernels carry no trace code.
int tpb_gemm_debug(int stages, int skip_mma);
int tpb_gemm_trace(int block);
int tpb_gemm_disable_flagged_exchange(int disable);
int tpb_gemm_enable_stream_k(int enable);
int tpb_gemm_trace_read(unsigned long long* out32);

#ifdef __cplusplus
}
#endif
