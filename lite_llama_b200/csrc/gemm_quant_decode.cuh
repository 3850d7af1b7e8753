// W4A16 projections of small decode batches (entries: gemm_quant.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gemm {

// shapes the kernel takes and is the faster one for
bool quant_decode_wanted(int64_t M, int64_t K, int64_t group);
// layout 0: the reference's tensors (table strides given), 1: repacked (b2l_w4a16_pack_*)
int quant_decode_gemm(int layout, void* y, int64_t ldy, const void* x, int64_t ldx, const void* w, int64_t ldw_words,
                      const float* scales, const float* zeros, int64_t s_stride_n, int64_t s_stride_k, const void* bias,
                      int bias_is_f32, int64_t M, int64_t N, int64_t K, int64_t group, int swiglu, int whole_zeros,
                      cudaStream_t st);

}  // namespace gemm
