// Results of the quantised pair GEMMs from registers to memory.  A lane holds one output (a weight row) of many tokens, in
// pairs of tokens; rows of Y are contiguous in the outputs.  Stores of two bytes per lane cover 64 bytes of one token, so a
// tile's end was bound by them; here lanes exchange packed values until each has four neighbouring outputs of one token.
#pragma once
#include "dequant.cuh"

namespace gemm {

#ifdef __CUDACC__

// four neighbouring outputs of a token, `left` of them in range
__device__ __forceinline__ void store4(__half* dst, uint2 v, int left, int vec) {
  if (vec && left >= 4) {
    *reinterpret_cast<uint2*>(dst) = v;
  } else {
    const __half* f = reinterpret_cast<const __half*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i < left) dst[i] = f[i];
  }
}
// p: {token t, t + 1} of this lane's output; even lanes of a pair (distance BIT) get token t of both outputs, odd ones t + 1
template <int BIT>
__device__ __forceinline__ uint32_t exchange_pair(uint32_t p, int lane) {
  return __byte_perm(p, __shfl_xor_sync(0xffffffffu, p, BIT), lane & BIT ? 0x3276u : 0x5410u);
}
// two words for the group whose bit BIT is clear, two for the other one: each lane keeps its own and gets its partner's
template <int BIT>
__device__ __forceinline__ uint2 exchange_word(uint32_t lo, uint32_t hi, int lane) {
  const bool up = lane & BIT;
  const uint32_t r = __shfl_xor_sync(0xffffffffu, up ? lo : hi, BIT);
  return up ? make_uint2(r, hi) : make_uint2(lo, r);
}
// a, b: {t, t + 1} and {t + 2, t + 3} of this lane's output -> token t + (lane & 3), outputs of lanes l & ~3 .. l | 3
__device__ __forceinline__ uint2 exchange4(uint32_t a, uint32_t b, int lane) {
  return exchange_word<2>(exchange_pair<1>(a, lane), exchange_pair<1>(b, lane), lane);
}
// SiLU(gate) * up, both already rounded to fp16 (gemm_quant.cu)
__device__ __forceinline__ float swiglu_h2(uint32_t gate_up) {
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&gate_up));
  return silu_q(f.x) * f.y;
}

// 2 NP tokens from row m0 of y on, `rows` of them in range; the warp's outputs start at n0 (a multiple of 32)
template <int NP>
__device__ __forceinline__ void store_rows(const uint64_t* acc, __half* y, int64_t ldy, int m0, int rows, int n0, int N, float bias,
                                           int lane, int vec) {
  const int col = n0 + (lane & ~3);
  __half* yp = y + (int64_t)(m0 + (lane & 3)) * ldy + col;
#pragma unroll
  for (int j = 0; j < NP; j += 2) {
    float f[4];
    unpack_f32x2(acc[j], f[0], f[1]);
    unpack_f32x2(acc[j + 1], f[2], f[3]);
    const uint2 v = exchange4(pack2<__half>(f[0] + bias, f[1] + bias), pack2<__half>(f[2] + bias, f[3] + bias), lane);
    if (2 * j + (lane & 3) < rows) store4(yp, v, N - col, vec);
    yp += 4 * ldy;
  }
}
// the same with SiLU(gate) * up over (gate_i, up_i) row pairs: eight tokens at a time, of two the even lane forms the first
// result and the odd lane the second; o0: the warp's first output (a multiple of 16), O: outputs
template <int NP>
__device__ __forceinline__ void store_swiglu(const uint64_t* acc, __half* y, int64_t ldy, int m0, int rows, int o0, int O, float bias,
                                             int lane, int vec) {
  const int col = o0 + ((lane & ~7) >> 1);
  __half* yp = y + (int64_t)(m0 + (lane & 7)) * ldy + col;
#pragma unroll
  for (int j = 0; j < NP; j += 4) {
    uint32_t d[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float o[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        float a, b;
        unpack_f32x2(acc[j + 2 * u + q], a, b);
        o[q] = swiglu_h2(exchange_pair<1>(pack2<__half>(a + bias, b + bias), lane));
      }
      d[u] = exchange_pair<2>(pack2<__half>(o[0], o[1]), lane);
    }
    const uint2 v = exchange_word<4>(d[0], d[1], lane);
    if (2 * j + (lane & 7) < rows) store4(yp, v, O - col, vec);
    yp += 8 * ldy;
  }
}

#endif  // __CUDACC__

}  // namespace gemm
