// Weight-only quantised GEMM for prompt-sized batches (entries: gemm_quant.cu).
#pragma once
#include <cuda_fp16.h>
#include "tma_desc.cuh"

namespace gemm {

struct QuantPairParams {
  void* y; int64_t ldy;                              // [M, N] fp16, or [M, N / 2] with the fused activation
  const void* bias; int bias_is_f32;
  const float* scales; int64_t s_stride_n, s_stride_k;
  int64_t s_stride_e;                                // grouped: expert stride
  const float* zeros;                                // int4: packed table
  int group_n;
  const int32_t* table;                              // grouped: {tiles, {expert, first row, rows} per tile}
  const int32_t* order;                              // grouped down projection: slot of every sorted row
  const __half* row_weights;                         // grouped down projection: routing weight by slot
  int M, N, steps, seg_steps, groups, m_tiles, n_tiles;      // filled by quant_pair_gemm (groups: pitch of the int4 tables)
  int vec;                                           // y in stores of four outputs
  int split_steps;                                   // a tile shared by several pairs: steps of each
  int tiles, split_from;                             // wide tiles: their number, and the first that is cut in two
};

// shapes the pair kernel takes and is the faster one for (see gemm_quant_pair.cu); qk: QuantKind
bool quant_pair_wanted(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k);
// pairs that share a tile, -1: tiles of 256 tokens, 0: not wanted
int quant_pair_form(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k, int swiglu);
int quant_pair_gemm(int qk, QuantPairParams& p, const void* x, int64_t ldx, const void* w, int64_t w_stride_bytes,
                    int64_t M, int64_t N, int64_t K, int64_t group_k, int swiglu, cudaStream_t st);
// the same with 256 tokens per tile (gemm_quant_wide.cu); boxes of the tensor maps: 128 weight rows, 64 tokens
bool quant_wide_wanted(int qk, int64_t M, int64_t N, int64_t steps, int64_t seg_steps, int swiglu);
int quant_wide_gemm(int qk, QuantPairParams& p, const CUtensorMap& tw, const CUtensorMap& tx, int swiglu, cudaStream_t st);

// The two products of a routed SwiGLU layer over activations sorted by expert (moe_routing.cu: b2l_moe_sort, b2l_moe_gather).
struct MoePairGemm {
  void* y; int64_t ldy;                              // gate_up: [rows, N / 2] sorted; down: [slots, N]
  const void* x; int64_t ldx;                        // [rows, K] sorted
  const void* w; int64_t w_row_stride;               // [experts, N, K] bytes
  const float* scales; int64_t s_stride_e, s_stride_n, s_stride_k;
  int64_t group_n, group_k;
  int64_t experts, rows, N, K;
  const int32_t* table; int64_t max_tiles; int tile_rows;
  const int32_t* order; const void* row_weights;     // down only
};

}  // namespace gemm
