// Weight-only quantised GEMM for prompt-sized batches (entries: gemm_quant.cu).
#pragma once
#include "tma_desc.cuh"

namespace gemm {

struct QuantPairParams {
  void* y; int64_t ldy;                              // [M, N] fp16, or [M, N / 2] with the fused activation
  const void* bias; int bias_is_f32;
  const float* scales; int64_t s_stride_n, s_stride_k;
  const float* zeros;                                // int4: packed table
  int group_n;
  int M, N, steps, seg_steps, m_tiles, n_tiles;      // filled by quant_pair_gemm
};

// shapes the pair kernel takes and is the faster one for (see gemm_quant_pair.cu); qk: QuantKind
bool quant_pair_wanted(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k);
int quant_pair_gemm(int qk, QuantPairParams& p, const void* x, int64_t ldx, const void* w, int64_t w_stride_bytes,
                    int64_t M, int64_t N, int64_t K, int64_t group_k, int swiglu, cudaStream_t st);

}  // namespace gemm
