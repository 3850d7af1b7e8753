// Weight-only quantised projections of decode batches: W4A16 (both layouts, the same bits) and W8A16, up to 64 tokens (entries:
// gemm_quant.cu; formats and reference lines there).
//
// Bound: HBM for 8-bit weights with many tiles (28672 x 4096, 32 tokens: 117 MB in 21.6 us, 5.4 TB/s), else latency: a 4096 x
// 4096 projection gives every SM 60 to 110 KB to read, convert and multiply, which takes less than the hand-offs around it.
// The streaming kernel (gemm_quant.cu) moves every block of weights from a loader to conversion warps, an MMA warp and drain
// warps, each hand-off a barrier between warps that wait for a turn on their scheduler.  Here
//   * three or four groups of four warps do everything for their own blocks (every NWG-th block of 128 rows x 128 bytes): a
//     thread converts its row into the group's operand columns of tensor memory, adds up the group's previous segment from
//     its accumulator columns, and has one barrier to wait for per 128 k (the products of that segment).  The groups run out
//     of step and hide one another's latencies; no sums leave a group before the tile ends.
//   * one helper warp per group issues its loads and its MMAs.  In the conversion warps these cost more than the conversion:
//     200 cycles for four MMAs, 450 for two activation loads of a 2900-cycle round (clock stamps, int4, 32 tokens).
//   * scales and zero points of repacked int4 travel with the block (2 KiB behind its 16), so a row's are two words of shared
//     memory; the others are loaded by the threads that use them, two blocks ahead.
//   * a tile's groups meet in tensor memory, where a row is the same lane for all of them: each group sums up some tokens.
//   * a tile shared by several CTAs is split evenly where possible, and every sharer then adds up its part of the tokens
//     (bq_plan): with one CTA reading all partial sums of 64 tokens, a 4096 x 4096 projection ended with 4 us of trips to L2.
//     The sharers then wait for one another, so all CTAs of a launch have to be resident at the same time: the grid is at most
//     one CTA per SM, and the calls of a device follow one another on one stream, as the workspace and the tickets that they have in
//     common demand in any case (kernels/_common.py).
//   * conversion starts before the previous kernel has ended (weights are static); only activations and results wait for it.
// Measured against the kernels that had these calls: quant_batch_wanted below.  Tried and not kept: both halves of a segment
// handed to the MMAs one by one (28672 x 4096, int4, 32 tokens 30 us), accumulators or operands in two buffers (three
// groups, 21.9; four groups with one buffer 18.0), the helpers split into loaders and issuers (fewer registers for the
// groups, 30), MMAs predicated on their lane instead of in a branch (+2 %).
// Numerics are the streaming kernel's: unscaled integer / e4m3 operands, whole zero points subtracted exactly, others (known
// only on the device in the reference's layout) as scale * (segment - z * sum of x), acc = fma(scale, segment, acc) in fp32; the sum over k runs over every NWG-th
// block first, then over groups and CTAs in a fixed order, with all 32 bits of every partial sum (bq_partial).
#define B2L_HANG_NORETURN true
#include "gemm_tc.cuh"
#include "dequant.cuh"
#include "gemm_quant_batch.cuh"
#include "gemm_quant_decode.cuh"

namespace gemm {

namespace {

constexpr int kBqStepK = 128;                                // k per accumulator segment
constexpr int kBqMaxW = 4, kBqMaxX = 8, kBqMaxGroups = 4;
// conversion groups: four, or the three that keep two activation stages of more than 32 tokens and 64 sums per thread
__host__ __device__ constexpr int bq_groups(int nt) { return nt <= 32 ? 4 : 3; }
constexpr int kBqCols = 128;                                 // tensor-memory columns of a group: operand (64), accumulator
__host__ __device__ constexpr int bq_threads(int nt) { return (bq_groups(nt) + 1) * 128; }
// registers per lane: 20 warps x 96 at launch = 16 x 104 + 4 x 64, 16 x 128 = 12 x 152 + 4 x 56
__host__ __device__ constexpr int bq_regs(int nt) { return bq_groups(nt) == 4 ? 104 : 152; }
__host__ __device__ constexpr int bq_helper_regs(int nt) { return bq_groups(nt) == 4 ? 64 : 56; }
// a raw block of weights, behind it its int4 tables: up to two groups of 128 scales and of 128 zero points (repacked), or four
// scales and four zero points of each row
__host__ __device__ constexpr int bq_slot_bytes(int qk, int layout) { return kABytes + (qk != Q_INT4 ? 0 : layout == 1 ? 2048 : 4096); }
// tensor maps of the reference's int4 tables
template <int QK, int LAYOUT> struct BqMaps {};
template <> struct BqMaps<Q_INT4, 0> { CUtensorMap s, z; };
__host__ __device__ constexpr int bq_x_bytes(int nt) { return 2 * nt * kStageKBytes; }
constexpr int kBqSmemMax = 227 * 1024 - 1024;
__host__ __device__ constexpr int bq_w_stages(int qk, int layout, int nt) {
  const int n = (kBqSmemMax / bq_groups(nt) - 2 * bq_x_bytes(nt)) / bq_slot_bytes(qk, layout);
  return n < kBqMaxW ? n : kBqMaxW;
}
__host__ __device__ constexpr int bq_x_stages(int qk, int layout, int nt) {
  const int left = kBqSmemMax / bq_groups(nt) - bq_w_stages(qk, layout, nt) * bq_slot_bytes(qk, layout);
  return left / bq_x_bytes(nt) < kBqMaxX ? left / bq_x_bytes(nt) : kBqMaxX;
}

struct __align__(8) BqControl {
  uint64_t w_full[kBqMaxGroups][kBqMaxW];    // a raw weight block has landed
  uint64_t x_full[kBqMaxGroups][kBqMaxX];
  uint64_t op_full[kBqMaxGroups];            // a segment of converted weights is in tensor memory, the previous one's sums are
                                             // out of it (4 warps)
  uint64_t done[kBqMaxGroups];               // a segment's products have retired
  uint32_t tmem_base;
};
static_assert(sizeof(BqControl) <= 1024, "control block too large");

__device__ __forceinline__ void bq_umma(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void bq_cp_async_4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ float bq_lds(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 bq_lds_128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
// A partial sum travels as one word that is not zero once it is there, all 32 bits of it: +0 goes as -0, which adds the same to
// a sum that starts at +0.
__device__ __forceinline__ uint32_t bq_partial(float f) {
  const uint32_t w = __float_as_uint(f);
  return w != 0u ? w : 0x80000000u;
}
// CTA that owns a raw block of the linearised (tile, raw block) space; 32 bits hold total * (ctas + 1) (host)
__host__ __device__ __forceinline__ int bq_owner(int lin, int ctas, int total) {
  return (int)((((unsigned)lin + 1u) * (unsigned)ctas - 1u) / (unsigned)total);
}

// LAYOUT (int4): 1 = the load-time repack, 0 = the reference's tensors (gemm_quant.cu)
template <int QK, int NT, int EPI, int LAYOUT>
__global__ void __launch_bounds__(bq_threads(NT), 1)
gemm_quant_batch_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                        const __grid_constant__ BqMaps<QK, LAYOUT> tabs, const QuantBatchParams p) {
  constexpr int NWG = bq_groups(NT), WS = bq_w_stages(QK, LAYOUT, NT), XS = bq_x_stages(QK, LAYOUT, NT);
  constexpr int kSlot = bq_slot_bytes(QK, LAYOUT), kX = bq_x_bytes(NT), kCols = kBqCols;
  constexpr int SEGS = QK == Q_INT4 ? 2 : 1;               // segments per raw block (128 rows x 128 bytes)
  static_assert(XS >= 2, "activation ring");
  extern __shared__ __align__(1024) uint8_t smem[];
  BqControl* ctl = reinterpret_cast<BqControl*>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // warps 0 .. 4 NWG - 1: conversion groups; then one helper per group: its loads and its MMAs
  const bool helper = warp >= 4 * NWG && (warp & 3) < NWG;
  const int wg = warp < 4 * NWG ? warp >> 2 : (warp & 3) < NWG ? warp & 3 : 0;
  uint8_t* w_ring = smem + 1024 + wg * (WS * kSlot + XS * kX);
  uint8_t* x_ring = w_ring + WS * kSlot;
  const int g0 = (int)((blockIdx.x * (unsigned)p.total) / (unsigned)p.ctas);
  const int g1 = (int)(((blockIdx.x + 1u) * (unsigned)p.total) / (unsigned)p.ctas);
  const int nblk = g1 - g0;

  // helper: raw block (tile, rb) into ring slot `slot`
  auto issue_w = [&](int tile, int rb, int slot) {
    uint8_t* dst = w_ring + slot * kSlot;
    uint64_t* bar = &ctl->w_full[wg][slot];
    if (QK == Q_INT4 && LAYOUT == 1) {
      // the scale groups that the block touches: two of 128 k, or one (two where a longer odd group ends inside)
      const bool tail = rb * 2 + 1 >= p.steps;
      int g_lo = rb * 2, cnt = tail ? 1 : 2;
      if (p.group_steps != 1) {
        g_lo = rb * 2 / p.group_steps;
        cnt = tail ? 1 : (rb * 2 + 1) / p.group_steps - g_lo + 1;
      }
      const uint32_t bytes = (uint32_t)cnt * kBlockW * 4;
      const int64_t src = ((int64_t)tile * p.groups + g_lo) * kBlockW;
      mbar_arrive_expect_tx(bar, kABytes + 2 * bytes);
      bulk_g2s(dst + kABytes, p.scales + src, bytes, bar);
      bulk_g2s(dst + kABytes + 1024, p.zeros + src, bytes, bar);
    } else if (QK == Q_INT4 && p.quads) {
      mbar_arrive_expect_tx(bar, kABytes + 4096);
      const int g = rb * 2 / p.group_steps & ~3;            // both steps' groups are in the same four (host)
      if constexpr (QK == Q_INT4 && LAYOUT == 0) {
        tma_load_2d(dst + kABytes, &tabs.s, g, tile * kBlockW, bar);
        tma_load_2d(dst + kABytes + 2048, &tabs.z, g, tile * kBlockW, bar);
      }
    } else {
      mbar_arrive_expect_tx(bar, kABytes);
    }
    tma_load_2d_hint(dst, &tmap_w, rb * (QK == Q_INT4 ? 32 : 128), tile * kBlockW, bar, kEvictFirst);
  };
  auto issue_x = [&](int step, int slot) {                 // activations of 128-k step `step`
    uint64_t* bar = &ctl->x_full[wg][slot];
    mbar_arrive_expect_tx(bar, kX);
    tma_load_2d_hint(x_ring + slot * kX, &tmap_x, step * kBqStepK, 0, bar, kEvictLast);
    tma_load_2d_hint(x_ring + slot * kX + kX / 2, &tmap_x, step * kBqStepK + 64, 0, bar, kEvictLast);
  };
  // the group's next weight request
  int w_tile = 0, w_rb = 0, w_i = wg;
  auto next_w = [&](int slot) {
    if (w_i < nblk) {
      if (elect_one()) issue_w(w_tile, w_rb, slot);
      __syncwarp();
      w_i += NWG;
      w_rb += NWG;
      while (w_rb >= p.nrb_tile) { w_rb -= p.nrb_tile; ++w_tile; }
    }
  };
  const int row = (warp & 3) * 32 + lane;
  // 8-bit scale of raw block i for this thread's row
  auto scale_of = [&](int i) {
    const int tile = (g0 + i) / p.nrb_tile, rb = g0 + i - tile * p.nrb_tile;
    int n = tile * kBlockW + row;
    n = n < p.N ? n : p.N - 1;
    return __ldg(p.scales + (int64_t)(n / p.group_n) * p.s_stride_n + (int64_t)(rb / p.group_steps) * p.s_stride_k);
  };
  float sc_next = 0.f, sc_next2 = 0.f;
  if (QK != Q_INT4 && warp < 4 * NWG) {
    if (wg < nblk) sc_next = scale_of(wg);
    if (wg + NWG < nblk) sc_next2 = scale_of(wg + NWG);
  }
  // the reference's int4 tables where they cannot be loaded four groups at a time: a thread copies its own row's scales of both
  // steps, and its zero points, behind the block
  int t_i = wg, t_rb = wg, t_tile = 0;                     // next block to copy for
  auto next_table = [&](int slot) {
    if (t_i < nblk) {
      const uint32_t dst = smem_u32(w_ring) + slot * kSlot + kABytes + row * 16;
      int n = t_tile * kBlockW + row;
      n = n < p.N ? n : p.N - 1;
      const int last = t_rb * 2 + 1 < p.steps ? 1 : 0;
      int g = t_rb * 2, g1 = g + last;
      if (p.group_steps != 1) { g /= p.group_steps; g1 /= p.group_steps; }
      const float* sp = p.scales + (int64_t)n * p.s_stride_n;
      const float* zp = p.zeros + (int64_t)n * p.s_stride_n;
      bq_cp_async_4(dst, sp + g * p.s_stride_k);
      bq_cp_async_4(dst + 4, sp + g1 * p.s_stride_k);
      bq_cp_async_4(dst + 2048, zp + g * p.s_stride_k);
      bq_cp_async_4(dst + 2048 + 4, zp + g1 * p.s_stride_k);
      t_i += NWG;
      t_rb += NWG;
      while (t_rb >= p.nrb_tile) { t_rb -= p.nrb_tile; ++t_tile; }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (QK == Q_INT4 && LAYOUT == 0 && !p.quads && warp < 4 * NWG) {
    t_tile = (g0 + wg) / p.nrb_tile;
    t_rb = g0 + wg - t_tile * p.nrb_tile;
    for (int s = 0; s < WS; ++s) next_table(s);
  }
  if (helper) {
    if (elect_one()) {
      for (int s = 0; s < WS; ++s) mbar_init(&ctl->w_full[wg][s], 1);
      mbar_fence_init();
      fence_proxy_async_smem();
    }
    __syncwarp();
    w_tile = (g0 + wg) / p.nrb_tile;
    w_rb = g0 + wg - w_tile * p.nrb_tile;
    // weights are static: requested before the previous kernel has finished
    for (int s = 0; s < WS; ++s) next_w(s);
    if (elect_one()) {
      for (int s = 0; s < XS; ++s) mbar_init(&ctl->x_full[wg][s], 1);
      mbar_init(&ctl->op_full[wg], 4);
      mbar_init(&ctl->done[wg], 1);
      mbar_fence_init();
      tma_prefetch_desc(&tmap_x);
    }
    __syncwarp();
  }
  if (warp == 0) {
    tmem_alloc(&ctl->tmem_base, 512);
    tmem_relinquish();
    pdl_launch_dependents();                               // after the allocation (gemm_dense.cu)
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t op_col = ctl->tmem_base + wg * kCols, acc_col = op_col + 64;

  if (warp >= 4 * NWG) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(bq_helper_regs(NT)));
    if (helper) {
      // ===================== helper: loads and MMAs of one group =====================
      constexpr uint32_t idesc = umma_idesc(1u, 0u, 0u, 0u, 0u, kBlockW, NT);
      const uint64_t x_desc0 = umma_desc_sw128_kmajor(smem_u32(x_ring));
      int rb = (g0 + wg) % p.nrb_tile;
      // next activation request: raw block, segment, slot
      int x_i = wg, x_rb = rb, x_seg = 0, x_to = 0;
      auto next_x = [&]() {
        if (x_i < nblk) {
          const int step = x_rb * SEGS + x_seg;
          if (elect_one()) issue_x(step, x_to);
          __syncwarp();
          if (++x_to == XS) x_to = 0;
          if (SEGS == 2 && x_seg == 0 && step + 1 < p.steps) {
            x_seg = 1;
          } else {
            x_seg = 0;
            x_i += NWG;
            x_rb += NWG;
            while (x_rb >= p.nrb_tile) x_rb -= p.nrb_tile;
          }
        }
      };
      pdl_wait_prior();                                    // the activations are the previous kernel's output
      for (int s = 0; s < XS; ++s) next_x();
      int x_slot = 0, w_slot = 0;
      uint32_t x_phase = 0, o_phase = 0;
      bool any = false;                                    // a segment has been issued
      for (int i = wg; i < nblk; i += NWG) {
        const int nseg = SEGS == 1 || rb * SEGS + SEGS <= p.steps ? SEGS : 1;
#pragma unroll 1
        for (int seg = 0; seg < nseg; ++seg) {
          const uint64_t b = x_desc0 + (uint64_t)(uint32_t)(x_slot * (kX >> 4));
          mbar_wait(&ctl->x_full[wg][x_slot], x_phase);
          mbar_wait(&ctl->op_full[wg], o_phase);
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              bq_umma(acc_col, op_col + 8 * j, b + (uint64_t)((j >> 2) * (kX / 2 >> 4) + 2 * (j & 3)), idesc, j != 0 ? 1u : 0u);
            tc_commit(&ctl->done[wg]);
          }
          __syncwarp();
          o_phase ^= 1;
          if (++x_slot == XS) { x_slot = 0; x_phase ^= 1; }
          // op_full: every word of the block has been converted, and the previous segment's products have retired
          if (seg == nseg - 1) next_w(w_slot);
          if (any) next_x();
          any = true;
        }
        if (++w_slot == WS) w_slot = 0;
        rb += NWG;
        while (rb >= p.nrb_tile) rb -= p.nrb_tile;
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(bq_regs(NT)));
    const int rx = row & 7;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    if (warp == 0) {
      // address translation of the workspace slots that this CTA reads at its very end (gemm_quant.cu)
      const int tile = (g1 - 1) / p.nrb_tile;
      const int c_lo = bq_owner(tile * p.nrb_tile, p.ctas, p.total), c_hi = bq_owner((tile + 1) * p.nrb_tile - 1, p.ctas, p.total);
      if ((p.even || c_lo == (int)blockIdx.x) && lane <= c_hi - c_lo && lane != (int)blockIdx.x - c_lo) {
        uint32_t d;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(d)
                     : "l"(p.ws + ((size_t)tile * p.slots + lane) * (NT * kBlockW)) : "memory");
      }
    }

    const uint32_t ring = smem_u32(w_ring);
    int w_slot = 0;
    uint32_t w_phase = 0, d_phase = 0;
    int x_slot = 0, x_prev = 0;                              // LAYOUT 0: activation stage of the segment
    uint32_t x_phase = 0, xp_prev = 0;
    int i = wg;
    for (int first = 0; first < nblk;) {
      const int tile = (g0 + first) / p.nrb_tile;
      int end = (tile + 1) * p.nrb_tile - g0;                // first raw block of the next tile
      end = end < nblk ? end : nblk;
      uint64_t acc[NT / 2];
#pragma unroll
      for (int j = 0; j < NT / 2; ++j) acc[j] = 0ull;
      bool pending = false;                                  // the previous segment has not been added up
      float sc_prev = 0.f, rest_prev = 0.f;

      auto drain = [&](float sc) {                           // acc += sc * segment
        if (QK == Q_INT4 && LAYOUT == 0 && __any_sync(0xffffffffu, rest_prev != 0.f)) {
          // zero points that cannot be folded into the conversion: acc += sc * (segment - z * sum of the activations), with the
          // segment's activations still in their stage.  Lane t sums up tokens t and t + 32
          mbar_wait(&ctl->x_full[wg][x_prev], xp_prev);
          float xs[2] = {0.f, 0.f};
#pragma unroll
          for (int u = 0; u < (NT + 31) / 32; ++u) {
            const int t = lane + 32 * u;
            if (t < NT) {
              const uint32_t src = smem_u32(x_ring) + x_prev * kX + t * 128;
#pragma unroll 4
              for (int c = 0; c < 16; ++c) {
                const uint4 v = bq_lds_128(src + (c >> 3) * (kX / 2) + (((c & 7) ^ (t & 7)) << 4));
                const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  const float2 f = __half22float2(h[q]);
                  xs[u] += f.x + f.y;
                }
              }
            }
          }
#pragma unroll
          for (int c = 0; c < NT; c += 16) {
            uint32_t pv[16];
            tmem_ld_32x32b_x16(acc_col + lane_off + c, pv);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              float a[2];
              unpack_f32x2(acc[(c + j) / 2], a[0], a[1]);
              const float x = __shfl_sync(0xffffffffu, xs[(c + j) >> 5], (c + j) & 31);
              a[j & 1] = fmaf(sc, fmaf(-rest_prev, x, __uint_as_float(pv[j])), a[j & 1]);
              acc[(c + j) / 2] = pack_f32x2(a[0], a[1]);
            }
          }
          return;
        }
        const uint64_t s2 = pack_f32x2(sc, sc);
        constexpr int CH = NT % 32 == 0 ? 32 : 16;
#pragma unroll
        for (int c = 0; c < NT; c += CH) {
          uint32_t pv[CH];
#pragma unroll
          for (int k = 0; k < CH; k += 16)
            tmem_ld_32x32b_x16(acc_col + lane_off + c + k, *reinterpret_cast<uint32_t(*)[16]>(pv + k));
          tc_wait_ld();
#pragma unroll
          for (int j = 0; j < CH / 2; ++j)
            acc[c / 2 + j] = fma_f32x2(s2, pack_f32x2(__uint_as_float(pv[2 * j]), __uint_as_float(pv[2 * j + 1])), acc[c / 2 + j]);
        }
      };
      for (; i < end; i += NWG) {
        const int rb = g0 + i - tile * p.nrb_tile;
        const float sc8 = sc_next;
        if (QK != Q_INT4) {
          sc_next = sc_next2;
          if (i + 2 * NWG < nblk) sc_next2 = scale_of(i + 2 * NWG);
        } else if (LAYOUT == 0 && !p.quads) {
          asm volatile("cp.async.wait_group %0;" ::"n"(WS - 1) : "memory");
        }
        mbar_wait(&ctl->w_full[wg][w_slot], w_phase);
        const uint32_t raw = ring + w_slot * kSlot;
        const int nseg = SEGS == 1 || rb * SEGS + SEGS <= p.steps ? SEGS : 1;
#pragma unroll 1
        for (int seg = 0; seg < nseg; ++seg) {
          float sc = sc8, rest = 0.f;
          __half2 add_lo, add_hi;
          constexpr int kChunks = QK == Q_INT4 ? 2 : 4;        // 16-byte chunks of the row per 64 k
          const uint32_t src = raw + row * 128;
          const int sx = (QK == Q_INT4 ? seg * 4 : 0) ^ rx;
          uint4 w[kChunks];
#pragma unroll
          for (int c = 0; c < kChunks; ++c) w[c] = bq_lds_128(src + ((sx ^ c) << 4));
          if (QK == Q_INT4) {
            float z;
            if (LAYOUT == 1) {
              uint32_t t = raw + kABytes + row * 4;
              if (seg != 0 && (p.group_steps == 1 || (rb * 2 + 1) % p.group_steps == 0)) t += kBlockW * 4;
              sc = bq_lds(t);
              z = bq_lds(t + 1024);
            } else {
              const int at = p.quads ? (rb * 2 + seg) / p.group_steps & 3 : seg;
              const uint32_t t = raw + kABytes + row * 16 + at * 4;
              sc = bq_lds(t);
              z = bq_lds(t + 2048);
              if (!(z >= 0.f && z <= 1023.f && z == rintf(z))) {
                rest = z;
                z = 0.f;
              }
            }
            add_lo = LAYOUT == 1 ? __float2half2_rn(-1024.f - z) : __floats2half2_rn(-1024.f - z, -64.f - z);
            add_hi = __float2half2_rn(-64.f - z);
          }
          uint32_t vals[32];
          auto convert = [&]() {
#pragma unroll
            for (int c = 0; c < kChunks; ++c) {
              const uint32_t ws[4] = {w[c].x, w[c].y, w[c].z, w[c].w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (QK == Q_INT4 && LAYOUT == 0) dequant_int4_word(ws[j], add_lo, vals + (QK == Q_INT4 ? 16 * c + 4 * j : 0));
                else if (QK == Q_INT4) dequant_int4_packed(ws[j], add_lo, add_hi, vals + (QK == Q_INT4 ? 16 * c + 4 * j : 0));
                else dequant_w8_word(ws[j], QK == Q_FP8, vals + (QK == Q_INT4 ? 0 : 8 * c + 2 * j));
              }
            }
          };
          convert();
          if (pending) {
            mbar_wait(&ctl->done[wg], d_phase);                // the previous segment
            d_phase ^= 1;
            tc_fence_after();
          }
          tmem_st_32x32b_x32(op_col + lane_off, vals);
#pragma unroll
          for (int c = 0; c < kChunks; ++c) w[c] = bq_lds_128(src + ((sx ^ (kChunks + c)) << 4));
          if (pending) drain(sc_prev);
          convert();
          tmem_st_32x32b_x32(op_col + lane_off + 32, vals);
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->op_full[wg]);
          sc_prev = sc;
          rest_prev = rest;
          if (QK == Q_INT4 && LAYOUT == 0) {
            x_prev = x_slot; xp_prev = x_phase;
            if (++x_slot == XS) { x_slot = 0; x_phase ^= 1; }
          }
          pending = true;
        }
        if (QK == Q_INT4 && LAYOUT == 0 && !p.quads) next_table(w_slot);
        if (++w_slot == WS) { w_slot = 0; w_phase ^= 1; }
      }
      if (pending) {
        mbar_wait(&ctl->done[wg], d_phase);
        d_phase ^= 1;
        tc_fence_after();
        drain(sc_prev);
      }
      // ---- the groups' sums meet in tensor memory (a row is the same lane for all of them) ----
      {
        uint32_t f[NT];
#pragma unroll
        for (int j = 0; j < NT / 2; ++j) {
          float a, b;
          unpack_f32x2(acc[j], a, b);
          f[2 * j] = __float_as_uint(a);
          f[2 * j + 1] = __float_as_uint(b);
        }
#pragma unroll
        for (int c = 0; c < NT; c += 16) tmem_st_32x32b_x16(acc_col + lane_off + c, f + c);
      }
      tc_wait_st();
      tc_fence_before();
      asm volatile("bar.sync 1, %0;" ::"n"(NWG * 128) : "memory");
      tc_fence_after();
      pdl_wait_prior();                                      // y and the workspace may still be in use upstream
      const int c_lo = bq_owner(tile * p.nrb_tile, p.ctas, p.total), c_hi = bq_owner((tile + 1) * p.nrb_tile - 1, p.ctas, p.total);
      const int slot = (int)blockIdx.x - c_lo, sharers = c_hi - c_lo + 1;
      const int n = tile * kBlockW + row;
      const bool n_ok = n < p.N;
      float bv = 0.f;
      if (n_ok && p.bias) bv = p.bias_is_f32 ? reinterpret_cast<const float*>(p.bias)[n]
                                             : __half2float(reinterpret_cast<const __half*>(p.bias)[n]);
      // sums of 8 tokens, in group order
      auto sum8 = [&](int c, float (&f)[8]) {
        uint32_t v[NWG][8];
#pragma unroll
        for (int u = 0; u < NWG; ++u) tmem_ld_32x32b_x8(ctl->tmem_base + u * kCols + 64 + lane_off + c * 8, v[u]);
        tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          f[e] = __uint_as_float(v[0][e]);
#pragma unroll
          for (int u = 1; u < NWG; ++u) f[e] += __uint_as_float(v[u][e]);
        }
      };
      auto store8 = [&](int c, const float (&f)[8]) {
        if (EPI == 0) {
          __half* yp = p.y + (int64_t)(c * 8) * p.ldy + n;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (n_ok && c * 8 + e < p.M) *yp = __float2half_rn(f[e] + bv);
            yp += p.ldy;
          }
        } else {
          // SiLU(gate) * up over (gate_i, up_i) row pairs, both rounded to fp16 first (gemm_quant.cu): of two tokens the
          // even lane forms the first result and the odd lane the second
          const bool odd = lane & 1;
          __half* yp = p.y + (int64_t)(c * 8 + (odd ? 1 : 0)) * p.ldy + (n >> 1);
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float a = __half2float(__float2half_rn(f[e] + bv)), b = __half2float(__float2half_rn(f[e + 1] + bv));
            const float other = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
            const float gate = odd ? other : a, up = odd ? b : other;
            if (n_ok && c * 8 + e + (odd ? 1 : 0) < p.M) *yp = __float2half_rn(silu_q(gate) * up);
            yp += 2 * p.ldy;
          }
        }
      };
      // Sharers that have no other tile (p.even) add up a part of the tokens each, else the first one all of them: the tile is
      // then the last of its range, and the tile that a later sharer has in common with it is the first of that one's.
      auto mine = [&](int c) { return p.even ? c % sharers == slot : slot == 0; };
      // a slot is [NT / 4][row][4 tokens]: 512 consecutive bytes per access of a warp
      uint4* base = reinterpret_cast<uint4*>(p.ws + (size_t)tile * p.slots * (NT * kBlockW)) + row;
      constexpr int kSlotVec = NT * kBlockW / 4, kChVec = kBlockW * 2;
#pragma unroll 1
      for (int c = wg; c < NT / 8; c += NWG) {
        if (sharers > 1 && mine(c)) continue;
        float f[8];
        sum8(c, f);
        if (sharers == 1) {
          store8(c, f);
        } else {
          uint32_t t[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) t[e] = bq_partial(f[e]);
          uint4* dst = base + slot * kSlotVec + c * kChVec;
          dst[0] = make_uint4(t[0], t[1], t[2], t[3]);
          dst[kBlockW] = make_uint4(t[4], t[5], t[6], t[7]);
        }
      }
      if (sharers > 1) {
#pragma unroll 1
        for (int c = wg; c < NT / 8; c += NWG) {
          if (!mine(c)) continue;
          // SB slots are requested together: one trip to L2, not one per slot
          constexpr int SB = 6;
          float own[8], f[8];
          sum8(c, own);
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = 0.f;
#pragma unroll 1
          for (int s0 = 0; s0 < sharers; s0 += SB) {
            uint32_t v[SB][8];
            unsigned long long t0 = 0ull;
            for (;;) {
              // A word that is 0 is still missing.  Two ways to say so; which one leaves the loop over the weights in better order is the
              // compiler's accident (28672 x 4096, 32 tokens, us, minimum / predicate: with the activation 19.7 / 19.1, the reference's
              // layout with zero points that are not whole 43.1 / 42.0, repacked 18.6 / 19.4).
              constexpr bool kPredicate = NT == 32 && (EPI == 1 || (QK == Q_INT4 && LAYOUT == 0));
              uint32_t least = 1u;
              bool all = true;
#pragma unroll
              for (int u = 0; u < SB; ++u) {
                const uint4* src = base + (s0 + u) * kSlotVec + c * kChVec;
#pragma unroll
                for (int e = 0; e < 8; e += 4) {
                  v[u][e] = v[u][e + 1] = v[u][e + 2] = v[u][e + 3] = 1u;                      // nothing to wait for
                  if (s0 + u < sharers && s0 + u != slot)
                    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(v[u][e]), "=r"(v[u][e + 1]), "=r"(v[u][e + 2]), "=r"(v[u][e + 3])
                                 : "l"(src + e / 4 * kBlockW) : "memory");
                }
              }
#pragma unroll
              for (int u = 0; u < SB; ++u)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  if (kPredicate) all = all && v[u][e] != 0u;
                  else least = min(least, v[u][e]);
                }
              if (kPredicate ? all : least != 0u) break;
              const unsigned long long now = b2l_globaltimer();
              if (t0 == 0ull) t0 = now;
              const unsigned long long lim = b2l_hang_ctl.limit_ns;
              if (lim != 0ull && now - t0 > lim)
                b2l_hang_stop((uint32_t)tile, (uint32_t)s0, b2l_file_hash(__FILE__), __LINE__, now - t0);
            }
            // in slot order, whoever adds
#pragma unroll
            for (int u = 0; u < SB; ++u) {
              if (s0 + u < sharers) {
                uint4* src = base + (s0 + u) * kSlotVec + c * kChVec;
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] += s0 + u == slot ? own[e] : __uint_as_float(v[u][e]);
                if (s0 + u != slot) src[0] = src[kBlockW] = make_uint4(0u, 0u, 0u, 0u);        // leave the workspace clean
              }
            }
          }
          store8(c, f);
        }
      }
      if (end < nblk) {
        tc_fence_before();
        asm volatile("bar.sync 1, %0;" ::"n"(NWG * 128) : "memory");      // read: the regions take the next tile's segments
        tc_fence_after();
      }
      first = end;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(ctl->tmem_base, 512);
}

struct BqPlan { int nt, ctas, even, slots, nrb_tile, n_tiles, total; };
int bq_tokens(int64_t M) { return M <= 16 ? 16 : M <= 32 ? 32 : M <= 48 ? 48 : 64; }
BqPlan bq_plan(int qk, int64_t M, int64_t N, int64_t K) {
  BqPlan pl;
  pl.nt = bq_tokens(M);
  pl.n_tiles = (int)cdiv64(N, kBlockW);
  pl.nrb_tile = (int)cdiv64(K, qk == Q_INT4 ? 256 : 128);
  pl.total = pl.n_tiles * pl.nrb_tile;
  // Equal splits of every tile where the tiles leave SMs over, a block or more for each conversion group; where that leaves
  // too many SMs idle (and with more tiles than SMs) equal shares of the whole, whose CTAs work on two tiles or more.  Counted
  // in raw blocks per CTA, a shared tile costs about two and a second one two more (4096 x 4096, int4, 32 tokens: 128 CTAs with
  // four blocks of one tile 6.1 us, 148 with 3.5 blocks of one or two tiles 7.9; 4096 x 14336: 11.8 and 13.4).
  const int sms = b2l_num_sms(), groups = bq_groups(pl.nt), most = (pl.nrb_tile + groups - 1) / groups;
  int splits = sms / pl.n_tiles;
  if (splits > most) splits = most;
  pl.ctas = pl.total < sms ? pl.total : sms;
  pl.even = splits > 0 && (splits == most || (pl.nrb_tile + splits - 1) / splits + (splits > 1 ? 2 : 0) <=
                                                 (pl.total + pl.ctas - 1) / pl.ctas + 4);
  if (pl.even) pl.ctas = pl.n_tiles * splits;
  // Most CTAs that can share a tile, in closed form (a loop over the tiles took 1 us of every call).
  const int least = pl.total / pl.ctas;                     // blocks of the shortest share
  pl.slots = pl.even ? splits : (pl.nrb_tile - 1 + least - 1) / least + 1;
  return pl;
}

template <int QK, int NT, int EPI, int LAYOUT>
int launch_bq(const CUtensorMap& tw, const CUtensorMap& tx, const BqMaps<QK, LAYOUT>& tabs, const QuantBatchParams& p,
              cudaStream_t st) {
  constexpr int smem = 1024 + bq_groups(NT) * (bq_w_stages(QK, LAYOUT, NT) * bq_slot_bytes(QK, LAYOUT) +
                                            bq_x_stages(QK, LAYOUT, NT) * bq_x_bytes(NT));
  static_assert(smem <= 227 * 1024, "shared memory");
  auto kern = gemm_quant_batch_kernel<QK, NT, EPI, LAYOUT>;
  static int configured[64] = {0};
  B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, smem, configured));
  b2l_launch(kern, dim3((unsigned)p.ctas), dim3(bq_threads(NT)), (size_t)smem, st, tw, tx, tabs, p);
  B2L_LAUNCH_CHECK();
  return B2L_OK;
}
template <int QK, int EPI, int LAYOUT>
int launch_nt(int nt, const CUtensorMap& tw, const CUtensorMap& tx, const BqMaps<QK, LAYOUT>& tabs, const QuantBatchParams& p,
              cudaStream_t st) {
  switch (nt) {
    case 16: return launch_bq<QK, 16, EPI, LAYOUT>(tw, tx, tabs, p, st);
    case 32: return launch_bq<QK, 32, EPI, LAYOUT>(tw, tx, tabs, p, st);
    case 48: return launch_bq<QK, 48, EPI, LAYOUT>(tw, tx, tabs, p, st);
    default: return launch_bq<QK, 64, EPI, LAYOUT>(tw, tx, tabs, p, st);
  }
}

}  // namespace

bool quant_batch_takes(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k) {
  if (M > 64 || (group_k % kBqStepK != 0 && group_k < K)) return false;
  if (qk == Q_INT4 && K % kBqStepK != 0) return false;      // the packed tables are read per 128 k
  const int64_t total = cdiv64(N, kBlockW) * cdiv64(K, qk == Q_INT4 ? 256 : 128);
  return total < (1 << 22);                                 // the kernel's range arithmetic is 32-bit: total * (ctas + 1)
}

// Against the kernels that had these calls, us, other -> this one.
// Streaming kernel (more than 8 tokens; fp8 in blocks, int4): 4096 x 4096, 32 tokens fp8 10.1 -> 6.7, int4 8.5 -> 6.1; 64 tokens
// 12.5 -> 7.8; 28672 x 4096, 32 tokens fp8 23.5 -> 21.6 (117 MB: the memory), int4 20.6 -> 18.5.  With 49 - 64 tokens only three
// conversion groups fit and 8-bit weights of more than one tile per SM take 5 % longer here (28672 x 4096: 26.8 / 28.3), int4
// does not (26.0 / 25.5; 37888 x 3584 with the activation 36.3 / 25.0).
// Pair kernel (one scale per row): 4096 x 4096 13 -> 5.5, 28672 x 4096 one token 38 -> 21, 64 tokens 26 / 28.
// Decode kernel (int4 up to 8 tokens): it keeps what it takes, in both layouts with the same bits.  It is the faster one where
// little is read (one / eight tokens: 4096 x 4096 3.8 and 5.1, here 5.3), not with long or uneven k (4096 x 14336 9.7 and 12.6,
// here 10.5; 37888 x 3584, 14 slices for 16 warps, 19.0 and 20.3, here 17.8).
// The reference's int4 layout: 4096 x 4096, 32 tokens 10.7 / 7.9, 28672 x 4096 25.2 / 25.7, 64 tokens 29.8 / 32.2; zero points
// that are not whole, 32 tokens 20 / 11 and 93 / 47.
bool quant_batch_wanted(int qk, int layout, int64_t M, int64_t N, int64_t K, int64_t group_k) {
  if (!quant_batch_takes(qk, M, N, K, group_k)) return false;
  const bool large = cdiv64(N, kBlockW) > b2l_num_sms();
  if ((qk != Q_INT4 || layout == 0) && M > 48 && large) return false;
  return qk != Q_INT4 || !quant_decode_wanted(M, K, group_k);
}

int64_t quant_batch_workspace_bytes(int qk, int64_t M, int64_t N, int64_t K) {
  const BqPlan pl = bq_plan(qk, M, N, K);
  return pl.slots > 1 ? (int64_t)pl.n_tiles * pl.slots * pl.nt * kBlockW * 4 : 0;
}

int quant_batch_gemm(int qk, int layout, QuantBatchParams& p, const void* x, int64_t ldx, const void* w, int64_t w_stride_bytes,
                     int64_t M, int64_t N, int64_t K, int64_t group_k, int swiglu, cudaStream_t st) {
  const BqPlan pl = bq_plan(qk, M, N, K);
  p.M = (int)M; p.N = (int)N;
  p.ctas = pl.ctas; p.even = pl.even; p.slots = pl.slots; p.nrb_tile = pl.nrb_tile; p.total = pl.total;
  p.steps = (int)cdiv64(K, kBqStepK);
  p.groups = group_k >= K ? 1 : (int)(K / group_k);
  p.group_steps = group_k >= K ? p.steps : (int)(group_k / kBqStepK);
  CUtensorMap tw, tx;
  int rc;
  if (qk == Q_INT4) rc = b2l_make_tmap_2d(&tw, w, TMA_I32, (uint64_t)N, (uint64_t)(K / 8), (uint64_t)w_stride_bytes, kBlockW, 32, true);
  else rc = b2l_make_tmap_2d(&tw, w, TMA_U8, (uint64_t)N, (uint64_t)K, (uint64_t)w_stride_bytes, kBlockW, 128, true);
  if (rc != B2L_OK) return rc;
  rc = b2l_make_tmap_2d(&tx, x, TMA_F16, (uint64_t)M, (uint64_t)K, (uint64_t)ldx * 2, (uint32_t)pl.nt, 64, true);
  if (rc != B2L_OK) return rc;
  if (qk == Q_INT4 && layout == 0) {
    // Tables by TMA where four groups of a row are 16 aligned bytes and the two steps of a block are in the same four; else by
    // the threads, whose 4-byte copies take as long as the conversion (28672 x 4096, 32 tokens: 31 us).
    BqMaps<Q_INT4, 0> tabs;
    memset(&tabs, 0, sizeof(tabs));
    // (Rows of a tensor map lie behind one another: expanded or overlapping tables are the threads'.)
    p.quads = p.groups % 4 == 0 && (p.group_steps & (p.group_steps - 1)) == 0 && p.s_stride_k == 1 && p.s_stride_n % 4 == 0 &&
              p.s_stride_n >= p.groups &&
              ((uintptr_t)p.scales | (uintptr_t)p.zeros) % 16 == 0;
    if (p.quads) {
      rc = b2l_make_tmap_2d(&tabs.s, p.scales, TMA_I32, (uint64_t)N, (uint64_t)p.groups, (uint64_t)p.s_stride_n * 4, kBlockW, 4, false);
      if (rc == B2L_OK)
        rc = b2l_make_tmap_2d(&tabs.z, p.zeros, TMA_I32, (uint64_t)N, (uint64_t)p.groups, (uint64_t)p.s_stride_n * 4, kBlockW, 4, false);
      if (rc != B2L_OK) return rc;
    }
    return launch_nt<Q_INT4, 0, 0>(pl.nt, tw, tx, tabs, p, st);
  }
  p.quads = 0;
  if (qk == Q_INT4) return swiglu ? launch_nt<Q_INT4, 1, 1>(pl.nt, tw, tx, {}, p, st) : launch_nt<Q_INT4, 0, 1>(pl.nt, tw, tx, {}, p, st);
  if (qk == Q_FP8) return launch_nt<Q_FP8, 0, 0>(pl.nt, tw, tx, {}, p, st);
  return launch_nt<Q_INT8, 0, 0>(pl.nt, tw, tx, {}, p, st);
}

}  // namespace gemm
