// Weight-only quantised projections of decode batches, up to 64 tokens (entries: gemm_quant.cu).
#pragma once
#include <cuda_fp16.h>
#include "tma_desc.cuh"

namespace gemm {

struct QuantBatchParams {
  __half* y; int64_t ldy;                            // [M, N], or [M, N / 2] with the fused activation
  const void* bias; int bias_is_f32;
  const float* scales; int64_t s_stride_n, s_stride_k;
  const float* zeros;                                // int4: packed table, or with the strides of the scales
  int group_n;
  uint32_t* ws;                                      // all-zero between launches (gemm_quant.cu)
  int M, N, ctas, even, slots, nrb_tile, steps, groups, group_steps, total, quads;      // filled by quant_batch_gemm
};

// shapes the kernel takes, and those that it is also the fastest one for; qk: QuantKind; layout (int4): 1 repacked, 0 the
// reference's tensors
bool quant_batch_takes(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k);
bool quant_batch_wanted(int qk, int layout, int64_t M, int64_t N, int64_t K, int64_t group_k);
int64_t quant_batch_workspace_bytes(int qk, int64_t M, int64_t N, int64_t K);
int quant_batch_gemm(int qk, int layout, QuantBatchParams& p, const void* x, int64_t ldx, const void* w, int64_t w_stride_bytes,
                     int64_t M, int64_t N, int64_t K, int64_t group_k, int swiglu, cudaStream_t st);

}  // namespace gemm
