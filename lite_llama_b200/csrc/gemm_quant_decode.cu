// W4A16 projections of small decode batches (up to 8 tokens), on the reference's tensors or the load-time repacked layout
// (formats and reference lines: gemm_quant.cu); the same bits from both.
//
// Bound: HBM; what stands in the way is latency and then the conversion (one token, 28672 x 4096: 52 % of the issue slots are
// used, and the warps that do not issue wait for their turn or the math pipe, not for memory; profiles/pair_gemm_ncu.txt).
// The streaming kernel (gemm_quant.cu) passes every 16 KiB of weights through three hand-offs (TMA -> conversion warps -> tensor memory -> MMA
// warp -> epilogue warps), 0.7 us per block and SM, after 2 us of set-up, and adds up shared tiles across CTAs: 7 - 20 us for
// projections that take 1.5 - 10 us to read.  With so few tokens the products are cheap enough for mma.sync, whose operands
// are registers, so here a warp does everything for its weights and hands over nothing but sums:
//   * a CTA owns whole strips of 16 weight rows; its 16 warps split k: warp w takes the slices w, w + 16, ... of 256 values.
//     No sums cross CTAs.
//   * a thread copies exactly the words that it converts (cp.async, a ring of four strips per warp, 108 KiB in flight per SM
//     without a barrier), starting before the previous kernel has finished (weights are static).
//   * k is assigned to the MMA's k positions so that a thread's 16 bytes of packed weights are its own A fragments of eight
//     MMAs and 16 bytes of an activation row are its B fragments of two: the activations of a slice stay in registers.
//   * one chain of 8 MMAs per 128 k, scaled into the fp32 sum like the other kernels' segments; whole zero points are
//     subtracted exactly in the conversion, others as scale * (sum - z * xsum).  (Nibbles as fp16 subnormals, with the zero point applied to the sums, need 5 instead of 9
//     instructions per word and measured the same, in chunks of four: 15.4 us against 16.3 us for 28672 x 4096, 5.5 against 5.0
//     us for 6144 x 4096, so the exact form stays.)
//   * after a chunk of strips the warps add up their sums through shared memory in warp order (deterministic); the next
//     chunk's weights are on their way meanwhile, and the other warps go on to them while some add (a second barrier right after
//     the sums costs 6 % of 28672 x 4096).
// Measured, one token, repacked layout, no activation, weights from memory, launches in a row, streaming kernel -> this one: 4096 x 4096
// 7.0 -> 4.4 us, 6144 x 4096 8.3 -> 5.6, 28672 x 4096 19.6 -> 15.9 (with the activation 16.1), 4096 x 14336 12.9 -> 9.8.  Copies by TMA (one lane instead of address arithmetic in all): 0.3 us slower to start, 4096 x
// 14336 at eight tokens 13.1 -> 15.5.
#include "common.cuh"
#include "dequant.cuh"
#include "gemm_quant_decode.cuh"

namespace gemm {

namespace {

constexpr int kDecWarps = 16, kDecThreads = kDecWarps * 32;
constexpr int kDecSlice = 256, kDecBlocks = kDecSlice / 128;       // k per slice, 128-k blocks in it
constexpr int kDecUnit = kDecBlocks * (1024 + 128);                // a strip's slice: words, then {16 scales, 16 zeros} per block
// CHUNK: strips whose sums a thread holds at a time; the warps meet once per chunk.  With twelve strips to a CTA or more, chunks of
// seven and a ring that is a strip shorter to make room for them (28672 x 4096, one / eight tokens, us: chunks of four 16.9 and 17.7,
// of seven 15.9 and 17.2, with the activation 17.6 and 19.1, 16.1 and 17.4); with one or two, chunks of two leave registers (4096 x 14336,
// eight tokens 13.1 -> 12.5); chunks of seven for few strips cost 5 - 10 % (6144 x 4096, eight tokens 7.0 / 7.3).
__host__ __device__ constexpr int dec_depth(int chunk) { return chunk > 4 ? 3 : 4; }

struct DecParams {
  __half* y; int64_t ldy;
  const void* bias; int bias_is_f32;
  const __half* x; int64_t ldx;
  const uint32_t* w; int64_t ldw;          // words
  const float* scales; const float* zeros; // LAYOUT 1: [tile of 128 rows][group][128], 0: [row][group] with these strides
  int64_t s_stride_n, s_stride_k;
  int M, N, K, strips, groups, group_shift;    // group of 128-k block b: b >> group_shift
};

__device__ __forceinline__ void cp_async_16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// D = A * B + 0
__device__ __forceinline__ void mma_f16_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  d[0] = d[1] = d[2] = d[3] = 0.f;
  mma_m16n8k16<__half>(d, a, b0, b1);
}

// WHOLE: the packer has seen that every zero point is an integer in [0, 1023] (the test costs 10 % where it has to be made:
// 28672 x 4096, one token, chunks of four, 17.9 against 16.3 us)
template <int LAYOUT, int EPI, bool WHOLE, int CHUNK>
__global__ void __launch_bounds__(kDecThreads, 1)
gemm_quant_decode_kernel(const DecParams p) {
  extern __shared__ __align__(128) uint8_t smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;              // MMA fragment coordinates
  constexpr int kDecDepth = dec_depth(CHUNK);
  uint8_t* ring = smem + warp * kDecDepth * kDecUnit;
  float4* red = reinterpret_cast<float4*>(smem + kDecWarps * kDecDepth * kDecUnit);   // [strip][warp][lane]
  pdl_launch_dependents();
  const int s_lo = (int)((int64_t)blockIdx.x * p.strips / gridDim.x);
  const int s_hi = (int)((int64_t)(blockIdx.x + 1) * p.strips / gridDim.x);

  // chunks of equal size
  const int chunks = (s_hi - s_lo + CHUNK - 1) / CHUNK;
  const int step = chunks > 0 ? (s_hi - s_lo + chunks - 1) / chunks : 1;
  const int slices = p.K / kDecSlice;
  const int mine = slices > warp ? (slices - warp - 1) / kDecWarps + 1 : 0;      // this warp's slices

  // the warp's units in order: chunks of `step` strips, inside a chunk all strips of a slice before the next slice
  int f_chunk = s_lo, f_slice = 0, f_strip = s_lo, f_slot = 0;
  auto issue = [&]() {
    if (mine > 0 && f_chunk < s_hi) {
      uint8_t* dst = ring + f_slot * kDecUnit;
      const int kb = (warp + f_slice * kDecWarps) * kDecBlocks;                // first 128-k block
      int r0 = f_strip * 16 + g, r1 = r0 + 8;                         // rows past N: any row, the result is not stored
      r0 = r0 < p.N ? r0 : p.N - 1;
      r1 = r1 < p.N ? r1 : p.N - 1;
      const uint32_t* w0 = p.w + (int64_t)r0 * p.ldw + kb * 16 + t * 4;
      const uint32_t* w1 = p.w + (int64_t)r1 * p.ldw + kb * 16 + t * 4;
      int rt = f_strip * 16 + (lane & 15);
      rt = LAYOUT == 1 || rt < p.N ? rt : p.N - 1;                    // packed tables are padded to whole tiles
      const float* tab = (lane < 16 ? p.scales : p.zeros) +
                         (LAYOUT == 1 ? (int64_t)(rt >> 7) * p.groups * 128 + (rt & 127) : rt * p.s_stride_n);
      const int64_t tab_k = LAYOUT == 1 ? 128 : p.s_stride_k;
#pragma unroll
      for (int b = 0; b < kDecBlocks; ++b) {
        cp_async_16(dst + b * 1024 + lane * 16, w0 + b * 16);
        cp_async_16(dst + b * 1024 + 512 + lane * 16, w1 + b * 16);
        cp_async_4(dst + kDecBlocks * 1024 + b * 128 + lane * 4, tab + ((kb + b) >> p.group_shift) * tab_k);
      }
      const int end = f_chunk + step < s_hi ? f_chunk + step : s_hi;
      if (++f_strip == end) {
        if (++f_slice == mine) { f_slice = 0; f_chunk += step; }
        f_strip = f_chunk;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++f_slot == kDecDepth) f_slot = 0;
  };
#pragma unroll
  for (int i = 0; i < kDecDepth - 1; ++i) issue();
  pdl_wait_prior();                                   // the activations are the previous kernel's output

  int slot = 0;
  int held = -1;                                      // slice whose activations are in xf
  uint4 xf[kDecBlocks][4];                            // token g, k 32 t + 8 j of each block
  float xs[kDecBlocks][2];                            // sum of the block's activations, tokens 2t and 2t + 1
  for (int chunk = s_lo; chunk < s_hi; chunk += step) {
    const int in_chunk = s_hi - chunk < step ? s_hi - chunk : step;
    float acc[CHUNK][4];
#pragma unroll
    for (int r = 0; r < CHUNK; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
    for (int sl = 0; sl < mine; ++sl) {
      if (held != sl) {                               // k up to 4096: one slice per warp, loaded once
        held = sl;
        const uint4* xp = reinterpret_cast<const uint4*>(p.x + (int64_t)g * p.ldx + (warp + sl * kDecWarps) * kDecSlice + 32 * t);
#pragma unroll
        for (int b = 0; b < kDecBlocks; ++b) {
#pragma unroll
          for (int j = 0; j < 4; ++j) xf[b][j] = g < p.M ? __ldcg(xp + b * 16 + j) : make_uint4(0u, 0u, 0u, 0u);
        }
        if (!WHOLE) {
          const uint32_t ones[4] = {0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u};
#pragma unroll
          for (int b = 0; b < kDecBlocks; ++b) {
            float sum[4];
            mma_f16_zero(sum, ones, xf[b][0].x, xf[b][0].y);
            mma_m16n8k16<__half>(sum, ones, xf[b][0].z, xf[b][0].w);
#pragma unroll
            for (int j = 1; j < 4; ++j) {
              mma_m16n8k16<__half>(sum, ones, xf[b][j].x, xf[b][j].y);
              mma_m16n8k16<__half>(sum, ones, xf[b][j].z, xf[b][j].w);
            }
            xs[b][0] = sum[0];
            xs[b][1] = sum[1];
          }
        }
      }
#pragma unroll
      for (int r = 0; r < CHUNK; ++r) {
        if (r < in_chunk) {
          issue();
          asm volatile("cp.async.wait_group %0;" ::"n"(kDecDepth - 1) : "memory");
          __syncwarp();                               // the tables were copied by other lanes
          const uint8_t* src = ring + slot * kDecUnit;
#pragma unroll
          for (int b = 0; b < kDecBlocks; ++b) {
            const float* tab = reinterpret_cast<const float*>(src + kDecBlocks * 1024 + b * 128);
            const float s0 = tab[g], s1 = tab[g + 8];
            float z0 = tab[16 + g], z1 = tab[24 + g];
            float rest0 = 0.f, rest1 = 0.f;           // zero points that cannot be folded into the conversion
            if (!WHOLE) {
              if (!(z0 >= 0.f && z0 <= 1023.f && z0 == rintf(z0))) { rest0 = z0; z0 = 0.f; }
              if (!(z1 >= 0.f && z1 <= 1023.f && z1 == rintf(z1))) { rest1 = z1; z1 = 0.f; }
            }
            const __half2 lo0 = __float2half2_rn(-1024.f - z0), hi0 = __float2half2_rn(-64.f - z0);
            const __half2 lo1 = __float2half2_rn(-1024.f - z1), hi1 = __float2half2_rn(-64.f - z1);
            const uint4 wa = lds_128(src + b * 1024 + lane * 16);
            const uint4 wb = lds_128(src + b * 1024 + 512 + lane * 16);
            const uint32_t a4[4] = {wa.x, wa.y, wa.z, wa.w}, b4[4] = {wb.x, wb.y, wb.z, wb.w};
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint32_t u[4], v[4];                    // k pairs (0,1) (2,3) (4,5) (6,7) of rows g and g + 8
              if (LAYOUT == 1) {
                dequant_int4_packed(a4[j], lo0, hi0, u);
                dequant_int4_packed(b4[j], lo1, hi1, v);
              } else {
                dequant_int4_word(a4[j], __lows2half2(lo0, hi0), u);
                dequant_int4_word(b4[j], __lows2half2(lo1, hi1), v);
              }
              const uint32_t f0[4] = {u[0], v[0], u[1], v[1]}, f1[4] = {u[2], v[2], u[3], v[3]};
              mma_m16n8k16<__half>(sum, f0, xf[b][j].x, xf[b][j].y);
              mma_m16n8k16<__half>(sum, f1, xf[b][j].z, xf[b][j].w);
            }
            if (!WHOLE && __any_sync(0xffffffffu, rest0 != 0.f || rest1 != 0.f)) {
#pragma unroll
              for (int c = 0; c < 4; ++c) sum[c] = fmaf(-(c < 2 ? rest0 : rest1), xs[b][c & 1], sum[c]);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(c < 2 ? s0 : s1, sum[c], acc[r][c]);
          }
          if (++slot == kDecDepth) slot = 0;
          __syncwarp();                               // every lane has read the tables before the slot is refilled
        }
      }
    }
    // ---- sums of the 16 warps, in warp order ----
    if (chunk != s_lo) __syncthreads();               // the last chunk's have been read
#pragma unroll
    for (int r = 0; r < CHUNK; ++r)
      if (r < in_chunk) red[(r * kDecWarps + warp) * 32 + lane] = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
    __syncthreads();
    if (warp < in_chunk) {                            // warp r stores strip r; lane is the fragment's
      float4 v = red[warp * kDecWarps * 32 + lane];
#pragma unroll
      for (int w = 1; w < kDecWarps; ++w) {
        const float4 o = red[(warp * kDecWarps + w) * 32 + lane];
        v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      }
      const float f[4] = {v.x, v.y, v.z, v.w};        // (row, m) (row, m + 1) (row + 8, m) (row + 8, m + 1)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int row = (chunk + warp) * 16 + g + (c >> 1) * 8, m = 2 * t + (c & 1);
        float bv = 0.f;
        if (p.bias && row < p.N) bv = p.bias_is_f32 ? reinterpret_cast<const float*>(p.bias)[row]
                                                    : __half2float(reinterpret_cast<const __half*>(p.bias)[row]);
        const __half own = __float2half_rn(f[c] + bv);
        if (EPI == 0) {
          if (row < p.N && m < p.M) p.y[(int64_t)m * p.ldy + row] = own;
        } else {
          // (gate_i, up_i) row pairs sit four lanes apart; both rounded to fp16 first (gemm_quant.cu)
          const float other = __shfl_xor_sync(0xffffffffu, __half2float(own), 4);
          if ((g & 1) == 0 && row < p.N && m < p.M)
            p.y[(int64_t)m * p.ldy + (row >> 1)] = __float2half_rn(silu_q(__half2float(own)) * other);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

template <int LAYOUT, int EPI, bool WHOLE, int CHUNK>
int launch_dec_chunk(const DecParams& p, cudaStream_t st) {
  constexpr int smem = kDecWarps * dec_depth(CHUNK) * kDecUnit + CHUNK * kDecWarps * 32 * 16;
  static_assert(smem <= 227 * 1024, "shared memory");
  auto kern = gemm_quant_decode_kernel<LAYOUT, EPI, WHOLE, CHUNK>;
  static int configured[64] = {0};
  B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, smem, configured));
  const int sms = b2l_num_sms();
  b2l_launch(kern, dim3((unsigned)(p.strips < sms ? p.strips : sms)), dim3(kDecThreads), (size_t)smem, st, p);
  B2L_LAUNCH_CHECK();
  return B2L_OK;
}
template <int LAYOUT, int EPI, bool WHOLE>
int launch_dec(const DecParams& p, cudaStream_t st) {
  const int sms = b2l_num_sms();
  if (p.strips <= 2 * sms) return launch_dec_chunk<LAYOUT, EPI, WHOLE, 2>(p, st);
  if constexpr (LAYOUT == 1)
    if (p.strips >= 12 * sms) return launch_dec_chunk<LAYOUT, EPI, WHOLE, 7>(p, st);
  return launch_dec_chunk<LAYOUT, EPI, WHOLE, 4>(p, st);
}

}  // namespace

// Up to 8 tokens (one MMA column block: two of them take 26 us for 28672 x 4096, where the streaming kernel takes 19.5).  k
// beyond 4096 means that a warp loads the activations of several slices for every chunk: 8 tokens of k 14336 still win
// (12.3 against 13.0 us), of k 18944 lose (15.4 against 14.1; 4 tokens 12.5).
bool quant_decode_wanted(int64_t M, int64_t K, int64_t group) {
  // whole slices of 256 k, groups of 128 * 2^n
  if (M > 8 || K % kDecSlice != 0 || group % 128 != 0 || M * K > 8 * 14336) return false;
  const int64_t q = group / 128;
  return (q & (q - 1)) == 0;
}

int quant_decode_gemm(int layout, void* y, int64_t ldy, const void* x, int64_t ldx, const void* w, int64_t ldw_words,
                      const float* scales, const float* zeros, int64_t s_stride_n, int64_t s_stride_k, const void* bias,
                      int bias_is_f32, int64_t M, int64_t N, int64_t K, int64_t group, int swiglu, int whole_zeros,
                      cudaStream_t st) {
  DecParams p;
  p.y = (__half*)y; p.ldy = ldy; p.bias = bias; p.bias_is_f32 = bias_is_f32;
  p.x = (const __half*)x; p.ldx = ldx; p.w = (const uint32_t*)w; p.ldw = ldw_words;
  p.scales = scales; p.zeros = zeros; p.s_stride_n = s_stride_n; p.s_stride_k = s_stride_k;
  p.M = (int)M; p.N = (int)N; p.K = (int)K;
  p.strips = (int)cdiv64(N, 16);
  p.groups = (int)(K / group);
  p.group_shift = 0;
  while ((128ll << p.group_shift) < group) ++p.group_shift;
  if (layout == 0) return launch_dec<0, 0, false>(p, st);
  if (whole_zeros) return swiglu ? launch_dec<1, 1, true>(p, st) : launch_dec<1, 0, true>(p, st);
  return swiglu ? launch_dec<1, 1, false>(p, st) : launch_dec<1, 0, false>(p, st);
}

}  // namespace gemm
