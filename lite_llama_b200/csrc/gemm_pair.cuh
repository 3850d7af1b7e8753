// Dense GEMM for prompt-sized batches (entry: gemm_dense.cu).
#pragma once
#include "tma_desc.cuh"

namespace gemm {

struct PairGemm {
  void* y; int64_t ldy;              // [M, N] fp16 / bf16
  const void* bias;                  // [N]: output dtype (kind 0) or fp32 (kind 1), nullable
  const float* a_scale;              // kind 1: [M]
  const float* b_scale;              // kind 1: [N]
  int64_t M, N, K;
  int64_t ldx, ldw;                  // row strides in elements
  const void* x; const void* w;
};

// whether the pair kernel takes the call and is the faster one (see gemm_pair.cu); kind 0: 16-bit, 1: int8 operands
bool pair_gemm_wanted(int kind, const PairGemm& g);
int pair_gemm(int kind, int dtype, const PairGemm& g, cudaStream_t st);

}  // namespace gemm
