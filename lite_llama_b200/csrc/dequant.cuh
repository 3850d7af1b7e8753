// Conversion of quantised weights to exact fp16 operands in tensor memory, shared by the quantised GEMMs.
#pragma once
#include "common.cuh"

namespace gemm {

enum QuantKind { Q_INT4 = 0, Q_FP8 = 1, Q_INT8 = 2 };

#ifdef __CUDACC__

// ---- dequantisers: packed weights -> fp16 pairs in K order (one 32-bit TMEM column per pair) ----
__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t mask, uint32_t orv) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(orv));  // (a & mask) | orv
  return r;
}
// one int32 word (8 nibbles) -> 4 half2 {n0,n1} {n2,n3} {n4,n5} {n6,n7}
__device__ __forceinline__ void dequant_int4_word(uint32_t w, __half2 add, uint32_t* out) {
  // byte j holds nibbles (2j, 2j+1).  Replicate the byte into both halves, keep nibble 2j in the low
  // half's mantissa and nibble 2j+1 (still shifted left by 4) in the high half's, OR in the fp16
  // exponent of 1024: low = 1024 + n0, high = 1024 + 16*n1; one HFMA2 maps both back to exact integers.
  const __half2 mul = __halves2half2(__float2half(1.0f), __float2half(0.0625f));
  // add = {-(1024 + z), -(64 + z)}: an integer zero point z is subtracted in the same (exact) HFMA2
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t rep = __byte_perm(w, w, 0x1111 * j);
    const uint32_t h = lop3_and_or(rep, 0x00F0000Fu, 0x64006400u);
    const __half2 v = __hfma2(*reinterpret_cast<const __half2*>(&h), mul, add);
    out[j] = *reinterpret_cast<const uint32_t*>(&v);
  }
}
__device__ __forceinline__ uint32_t cvt_e4m3x2_f16x2(uint16_t v) {
  uint32_t r;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(r) : "h"(v));
  return r;
}
// one 32-bit word (4 bytes) -> 2 half2
__device__ __forceinline__ void dequant_w8_word(uint32_t w, bool fp8, uint32_t* out) {
  if (fp8) {
    out[0] = cvt_e4m3x2_f16x2((uint16_t)(w & 0xFFFFu));
    out[1] = cvt_e4m3x2_f16x2((uint16_t)(w >> 16));
  } else {
    // b -> u = b + 128 (xor 0x80), fp16(0x6400 | u) = 1024 + u, minus 1152 = b   (all exact)
    const __half2 off = __float2half2_rn(-1152.0f);
    const uint32_t u = w ^ 0x80808080u;
    const uint32_t h0 = __byte_perm(u, 0x64646464u, 0x4140u);   // [0x64, byte1, 0x64, byte0]
    const uint32_t h1 = __byte_perm(u, 0x64646464u, 0x4342u);
    const __half2 v0 = __hadd2(*reinterpret_cast<const __half2*>(&h0), off);
    const __half2 v1 = __hadd2(*reinterpret_cast<const __half2*>(&h1), off);
    out[0] = *reinterpret_cast<const uint32_t*>(&v0);
    out[1] = *reinterpret_cast<const uint32_t*>(&v1);
  }
}

// one repacked int4 word (b2l_w4a16_pack_qweight: nibble positions hold K indices [0,2,4,6,1,3,5,7]): each LOP3 yields a
// K-consecutive pair; low-nibble pairs are 1024 + n, high-nibble pairs 1024 + 16 n.  add_lo = {-(1024 + z)} x 2, add_hi =
// {-(64 + z)} x 2.  5 ALU-pipe instructions per word instead of 8.
__device__ __forceinline__ void dequant_int4_packed(uint32_t w, __half2 add_lo, __half2 add_hi, uint32_t* out) {
  const __half2 one = __float2half2_rn(1.0f), sixteenth = __float2half2_rn(0.0625f);
  const uint32_t w8 = w >> 8;
  const uint32_t h0 = lop3_and_or(w, 0x000F000Fu, 0x64006400u);
  const uint32_t h1 = lop3_and_or(w, 0x00F000F0u, 0x64006400u);
  const uint32_t h2 = lop3_and_or(w8, 0x000F000Fu, 0x64006400u);
  const uint32_t h3 = lop3_and_or(w8, 0x00F000F0u, 0x64006400u);
  const __half2 v0 = __hfma2(*reinterpret_cast<const __half2*>(&h0), one, add_lo);
  const __half2 v1 = __hfma2(*reinterpret_cast<const __half2*>(&h1), sixteenth, add_hi);
  const __half2 v2 = __hfma2(*reinterpret_cast<const __half2*>(&h2), one, add_lo);
  const __half2 v3 = __hfma2(*reinterpret_cast<const __half2*>(&h3), sixteenth, add_hi);
  out[0] = *reinterpret_cast<const uint32_t*>(&v0);
  out[1] = *reinterpret_cast<const uint32_t*>(&v1);
  out[2] = *reinterpret_cast<const uint32_t*>(&v2);
  out[3] = *reinterpret_cast<const uint32_t*>(&v3);
}

// registers -> TMEM: lane of the warp writes its own TMEM lane, 32 consecutive 32-bit columns
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ uint64_t pack_f32x2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
// two IEEE fused multiply-adds in one instruction
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm volatile("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// the swiglu kernel's SiLU (csrc/elementwise.cu), so the fused epilogue rounds like the unfused path
__device__ __forceinline__ float silu_q(float x) { return __fdividef(x, 1.0f + __expf(-x)); }
__device__ __forceinline__ uint4 lds_128(const void* p) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(smem_u32(p)));
  return v;
}

#endif  // __CUDACC__

}  // namespace gemm
