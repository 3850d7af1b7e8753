// Weight-only quantised GEMMs of prompt-sized batches on CTA pairs: W4A16 on the load-time repacked layout and W8A16
// (entries: gemm_quant.cu; formats and reference lines there).
//
// Bound: the tensor pipe, if the conversion of the weights keeps out of its way.  The streaming kernel (gemm_quant.cu)
// converts every weight tile once per 64 tokens; 128 weights x 128 k cost each scheduler ~190 issue slots to convert and
// 64 tokens of MMAs last 256 cycles, so its hand-offs were the critical path (430 - 500 TF/s).  Here the tile is 256
// weight rows x 128 tokens on a pair of SMs:
//   * 128 rows x 128 k feed 512 cycles of MMAs per SM: conversion (two groups of four warps, each its own half of the
//     operand stages) plus the drain of one accumulator segment take half of the issue slots: what was left was waiting at
//     hand-offs, most of all for the one issuing warp and for the trip of an accumulator (gemm_quant_wide.cu), so there are two
//     issuers and three or four accumulators where every 128 k are a segment of their own;
//   * cta_group::2: each SM stages 64 of the 128 tokens, 48 bytes per clock and SM from L2 for int4 weights;
//   * the operand stays in tensor memory beside the accumulators;
//   * a segment's buffer is handed back as soon as its columns are in the registers of eight epilogue warps, before the last
//     multiply-adds: with four warps that read it in two turns the MMAs waited for the drain (977 us against 900);
//   * the grid is persistent, rings run on across tiles.
// Measured, 28672 x 4096 at 4096 tokens, launches by themselves (streaming kernel -> this one; 15 - 20 % more in a pass that
// keeps the card at its power cap): int4 1853 -> 900 us (1.07 PFLOP/s), fp8 in 128 x 128
// blocks 1748 -> 867 us, int8 per channel 3124 -> 754 us (no drain before the end of k: 1.28 PFLOP/s).  A third accumulator
// at the cost of two operand stages: int4 878, fp8 901 us.  Sizes of that order are now taken by the kernel of 256 tokens per
// tile (gemm_quant_wide.cu), but for 8-bit weights in groups of 128 (fp8 in blocks 872 us in launches in a row, with 256 tokens 910).  One issuer and two accumulators -> two and three or four, us: int4 28672 x 4096 with the
// activation at 128 tokens 42.7 -> 36.8, 4096 x 14336 at 512 63 -> 54, fp8 in blocks 4096 x 4096 at 512 19.3 -> 17.1; experts (128 of
// 2048 x 768, fp8, top 8) gate|up and down at 2000 tokens 173 + 153 -> 135 + 126, at 32 69 + 46 -> 58 + 33.
// Numerics are the streaming kernel's: unscaled integer / e4m3 operands, zero points subtracted exactly, one segment of
// the accumulator per scale group, acc = fma(scale, segment, acc) in fp32 in ascending k.
#define B2L_HANG_NORETURN true   // common.cuh: 128 accumulators beside the wait loops
#include "gemm_tc.cuh"
#include "gemm_quant_pair.cuh"
#include "pair.cuh"
#include "dequant.cuh"
#include "gemm_quant_out.cuh"

namespace gemm {

constexpr int kQpThreads = 20 * 32;
constexpr int kQpWStages = 6, kQpXStages = 6, kQpMaxAcc = 4, kQpMaxOp = 8;
constexpr int kQpTokens = 128;                              // per pair tile; each CTA stages half
// Accumulators and operand steps that share tensor memory, for tiles of NT tokens.  Where every step of 128 k is a segment of
// its own, the trip of an accumulator (commit, wake-up, loads of the epilogue, arrival, issue: about 1000 cycles, the MMAs of a
// step 512 or 300) asks for three or four, and two issuing warps take turns.  CHAIN (longer segments): an accumulator's MMAs
// follow one another, so one warp issues them, and what a step waits for is its conversion: two accumulators, more steps.
__host__ __device__ constexpr int qp_accs(int nt, bool chain) { return chain ? 2 : nt == kQpTokens ? 3 : 4; }
__host__ __device__ constexpr int qp_op_steps(int nt, bool chain) { return (512 - qp_accs(nt, chain) * nt) / 64; }
constexpr int kQpStepK = 128;                               // k per operand step; handed over and back in stages of 64 where there are two steps of it
constexpr int kQpXSub = kQpTokens / 2 * kStageKBytes;       // 64 tokens x 64 k
constexpr int kQpXBytes = 2 * kQpXSub;
constexpr int kQpMeta = 8 * 64 * 8;                         // down projection: {slot, routing weight} of the epilogue warps' rows
constexpr int kQpSmem = 1024 + 1024 + kQpWStages * kABytes + kQpXStages * kQpXBytes + kQpMeta;
constexpr int kQpBand = 16;
constexpr int kQpEpi0 = 8, kQpWProd = 16, kQpXProd = 17, kQpMma = 18;   // eight conversion, eight epilogue warps, two issuers

struct __align__(8) QpControl {
  uint64_t w_full[kQpWStages];      // own: a raw weight block has landed
  uint64_t w_empty[kQpWStages];     // own: its words have been converted (4 warp arrivals per operand stage in it)
  uint64_t x_full[kQpXStages];      // leader: both CTAs' token halves have landed
  uint64_t x_empty[kQpXStages];     // both: the MMAs that read them have retired
  uint64_t op_full[kQpMaxOp];       // leader: both CTAs' converted rows are in tensor memory (8 warp arrivals)
  uint64_t op_empty[kQpMaxOp];      // both
  uint64_t acc_full[kQpMaxAcc];     // both: a segment is complete
  uint64_t acc_empty[kQpMaxAcc];    // leader: both CTAs' epilogue warps have read it (16 warp arrivals)
  uint32_t tmem_base;
};
static_assert(sizeof(QpControl) <= 1024, "control block too large");

// What a tile is: `mode` plain = one weight matrix; grouped = experts, one entry of the tile table per 128 rows of an
// expert's run of the sorted activations (moe_sort, moe_routing.cu), the entries' output tiles next to one another so that
// the pairs in flight share the activations and an expert's second entry finds the weights in L2.  The table and the slot
// order are earlier kernels' output, and this one may be resident before they are written: never read as data that is
// constant for the kernel (__ldg).
enum { QP_PLAIN = 0, QP_GATE_UP = 1, QP_DOWN = 2 };
struct QpTile { int n, m0, rows, expert; };
template <int MODE>
__device__ __forceinline__ int qp_tiles(const QuantPairParams& p) {
  return MODE == QP_PLAIN ? p.m_tiles * p.n_tiles : ld_upstream(p.table) * p.n_tiles;
}
template <int MODE>
__device__ __forceinline__ QpTile qp_tile(const QuantPairParams& p, int t) {
  QpTile o;
  if (MODE == QP_PLAIN) {
    const PairTile pt = pair_tile(t, p.m_tiles, p.n_tiles, kQpBand);
    o.n = pt.n; o.m0 = pt.m * kQpTokens; o.rows = p.M - o.m0; o.expert = 0;
  } else {
    const int e = t / p.n_tiles;
    o.n = t - e * p.n_tiles;
    o.expert = ld_upstream(p.table + 1 + 3 * e); o.m0 = ld_upstream(p.table + 2 + 3 * e); o.rows = ld_upstream(p.table + 3 + 3 * e);
  }
  return o;
}

// tokens of a tile rounded up to what cta_group::2 takes as N
template <int NT>
__device__ __forceinline__ int qp_tile_n(int rows_left) {
  const int n = (rows_left + 31) & ~31;
  return n < NT ? n : NT;
}

template <int QK, int EPI, int MODE, int NT, bool CHAIN, int S>
__global__ void __cluster_dims__(2 * S, 1, 1) __launch_bounds__(kQpThreads, 1)
gemm_quant_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                       const QuantPairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  QpControl* ctl = reinterpret_cast<QpControl*>(smem);
  uint8_t* w_ring = smem + 1024;
  uint8_t* x_ring = w_ring + kQpWStages * kABytes;
  constexpr int kHalf = NT / 2;                            // tokens per epilogue warp
  constexpr int kAccs = qp_accs(NT, CHAIN), kOpSteps = qp_op_steps(NT, CHAIN), kOpCol0 = kAccs * NT;
  constexpr int kSub = CHAIN || NT != kQpTokens ? 1 : 2, kOpStages = kSub * kOpSteps;      // stages per operand step
  // (plain mode with NT 64 is launched for up to 64 tokens only: one row of tiles)
  constexpr int kStepsPerRaw = QK == Q_INT4 ? 2 : 1;       // a raw block is 128 rows x 128 bytes

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // S > 1: S pairs share a tile and run over a part of k each (one tile per cluster)
  const uint32_t first = S > 1 ? pair_rank() & ~1u : 0u, rank = pair_rank() - first;
  const int pairs = gridDim.x / (2 * S), pair = blockIdx.x / (2 * S);
  auto lead = [&](const void* q) { return S > 1 ? cluster_addr(q, first) : leader_addr(q); };
  auto commit = [&](uint64_t* bar) {
    if (S > 1) tc_commit_pair_at(bar, first);
    else tc_commit_pair(bar);
  };
  if (MODE != QP_PLAIN) pdl_wait_prior();                  // the tile table is an earlier kernel's output
  const int tiles = qp_tiles<MODE>(p);
  const int step0 = S > 1 ? (int)(first / 2) * p.split_steps : 0;
  const int steps = S > 1 && p.steps - step0 > p.split_steps ? p.split_steps : p.steps - step0;      // operand steps of this pair
  if (threadIdx.x == kQpWProd * 32) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < kQpWStages; ++s) {
      mbar_init(&ctl->w_full[s], 1);
      mbar_init(&ctl->w_empty[s], 4 * kStepsPerRaw);
    }
    for (int s = 0; s < kQpXStages; ++s) {
      mbar_init(&ctl->x_full[s], 1);
      mbar_init(&ctl->x_empty[s], 1);
    }
    for (int s = 0; s < kOpStages; ++s) {
      mbar_init(&ctl->op_full[s], 8);
      mbar_init(&ctl->op_empty[s], 1);
    }
    for (int s = 0; s < kAccs; ++s) {
      mbar_init(&ctl->acc_full[s], 1);
      mbar_init(&ctl->acc_empty[s], 16);
    }
    mbar_fence_init();
  }
  if (warp == kQpMma) {
    tmem_alloc_pair(&ctl->tmem_base, 512);
    tmem_relinquish_pair();
    pdl_launch_dependents();        // after the allocation (gemm_dense.cu)
  }
  tc_fence_before();
  pair_sync();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  // registers per lane: five warpgroups x 96 at launch = 2 x 80 + 2 x 136 + 48 = 2 x 80 + 2 x 128 + 64 = 2 x 88 + 2 x 112 + 80
  constexpr bool kTall = NT == kQpTokens;
  constexpr int kRegsEpi = CHAIN ? 136 : kTall ? 128 : 112, kRegsConv = CHAIN ? 80 : kTall ? 80 : 88, kRegsRest = CHAIN ? 48 : kTall ? 64 : 80;
  if (warp >= kQpWProd) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsRest));
    if (warp == kQpWProd) {
      // ===================== raw weight blocks of this CTA's 128 rows =====================
      PipeState ws(kQpWStages);
      const int raws = (steps + kStepsPerRaw - 1) / kStepsPerRaw;
      for (int t = pair; t < tiles; t += pairs) {
        const QpTile pt = qp_tile<MODE>(p, t);
        const int row = MODE == QP_GATE_UP ? pt.expert * p.N + pt.n * kBlockW + (int)rank * (kBlockW / 2)
                                           : pt.expert * p.N + pt.n * 2 * kBlockW + (int)rank * kBlockW;
        for (int rb = 0; rb < raws; ++rb) {
          mbar_wait(&ctl->w_empty[ws.stage], ws.phase ^ 1);
          if (elect_one()) {
            mbar_arrive_expect_tx(&ctl->w_full[ws.stage], kABytes);
            uint8_t* dst = w_ring + (size_t)ws.stage * kABytes;
            const int col = (step0 / kStepsPerRaw + rb) * (QK == Q_INT4 ? 32 : 128);
            if (MODE == QP_GATE_UP) {
              // 16 gate rows, the 16 up rows of the same outputs, 16 gate rows ...: a warp then holds both
#pragma unroll
              for (int b = 0; b < 8; ++b)
                tma_load_2d_hint(dst + b * 16 * kStageKBytes, &tmap_w, col, row + (b & 1) * (p.N / 2) + (b >> 1) * 16,
                                 &ctl->w_full[ws.stage], kEvictNormal);
            } else {
              tma_load_2d_hint(dst, &tmap_w, col, row, &ctl->w_full[ws.stage], kEvictNormal);
            }
          }
          __syncwarp();
          ws.advance();
        }
      }
    } else if (warp == kQpXProd) {
      // ===================== activations: this CTA's half of the tile's tokens =====================
      pdl_wait_prior();
      PipeState xs(kQpXStages);
      for (int t = pair; t < tiles; t += pairs) {
        const QpTile pt = qp_tile<MODE>(p, t);
        const int half = qp_tile_n<NT>(pt.rows) / 2;            // rows of this CTA that the MMAs read
        const int row = pt.m0 + (int)rank * half;
        for (int s = 0; s < steps; ++s) {
          mbar_wait(&ctl->x_empty[xs.stage], xs.phase ^ 1);
          if (elect_one()) {
            uint8_t* dst = x_ring + (size_t)xs.stage * kQpXBytes;
            const uint32_t bar = lead(&ctl->x_full[xs.stage]);
            if (MODE == QP_PLAIN) {
              if (rank == 0) mbar_arrive_expect_tx(&ctl->x_full[xs.stage], 2 * kQpXBytes);
              tma_load_2d_pair(dst, &tmap_x, (step0 + s) * kQpStepK, row, bar, kEvictNormal);
              tma_load_2d_pair(dst + kQpXSub, &tmap_x, (step0 + s) * kQpStepK + 64, row, bar, kEvictNormal);
            } else {
              // an expert may have two rows: only the 16-row boxes that are read
              if (rank == 0) mbar_arrive_expect_tx(&ctl->x_full[xs.stage], 2 * 2 * half * kStageKBytes);
              for (int r = 0; r < half; r += 16) {
                tma_load_2d_pair(dst + r * kStageKBytes, &tmap_x, s * kQpStepK, row + r, bar, kEvictNormal);
                tma_load_2d_pair(dst + kQpXSub + r * kStageKBytes, &tmap_x, s * kQpStepK + 64, row + r, bar, kEvictNormal);
              }
            }
          }
          __syncwarp();
          xs.advance();
        }
      }
      // every stage handed back: no commit is still on its way to this CTA's barriers when it leaves
      for (int s = 0; s < kQpXStages; ++s) {
        mbar_wait(&ctl->x_empty[xs.stage], xs.phase ^ 1);
        xs.advance();
      }
    } else if (rank == 0 && (warp == kQpMma || !CHAIN)) {
      // ===================== MMA issuers (leader) =====================
      // Waits, 8 MMAs and commits of a step take a warp some 800 cycles, so two take turns where every step is a segment of its
      // own.  An operand stage and a slot of X are then always the same one's (both rings have an even number of steps), and of
      // an accumulator, whose turns alternate, the trip before the last one is over: the one after it was waited for at this
      // issuer's last step.
      static_assert(kOpSteps % 2 == 0 && kQpXStages % 2 == 0, "rings and issuers");
      const uint64_t x_desc0 = umma_desc_sw128_kmajor(smem_u32(x_ring));
      PipeState xs(kQpXStages), os(kOpSteps), as(kAccs);
      int turn = warp - kQpMma;                            // 0: the next step is this issuer's
      for (int t = pair; t < tiles; t += pairs) {
        const QpTile pt = qp_tile<MODE>(p, t);
        const uint32_t idesc = umma_idesc(1u, 0u, 0u, 0u, 0u, 2 * kBlockW, (uint32_t)qp_tile_n<NT>(pt.rows));
        int in_seg = 0;
        for (int s = 0; s < steps; ++s) {
          const bool last = !CHAIN || in_seg + 1 == p.seg_steps || s + 1 == steps;
          if (CHAIN || turn == 0) {
            const uint32_t acc = tmem_base + as.stage * NT, a = tmem_base + kOpCol0 + os.stage * 64;
            const uint64_t b = x_desc0 + (uint64_t)((xs.stage * kQpXBytes) >> 4);
            if (CHAIN && in_seg == 0) mbar_wait(&ctl->acc_empty[as.stage], as.phase ^ 1);
            mbar_wait(&ctl->x_full[xs.stage], xs.phase);
            mbar_wait(&ctl->op_full[kSub * os.stage], os.phase);
            if (!CHAIN) mbar_wait(&ctl->acc_empty[as.stage], as.phase ^ 1);
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < kSub; ++h) {
              if (h == 1) {
                mbar_wait(&ctl->op_full[kSub * os.stage + 1], os.phase);
                tc_fence_after();
              }
              if (elect_one()) {
#pragma unroll
                for (int k = h * 4; k < (kSub == 1 ? 8 : h * 4 + 4); ++k)
                  umma_pair_ts(acc, a + 8 * k, b + (uint64_t)((k >> 2) * (kQpXSub >> 4) + 2 * (k & 3)), idesc,
                               (in_seg | k) != 0 ? 1u : 0u);
                commit(&ctl->op_empty[kSub * os.stage + h]);
                if (h == kSub - 1) {
                  if (last) commit(&ctl->acc_full[as.stage]);
                  commit(&ctl->x_empty[xs.stage]);   // the last one: the X producers wait for it before they leave
                }
              }
              __syncwarp();
            }
          }
          if (!CHAIN) turn ^= 1;
          if (last) { as.advance(); in_seg = 0; } else { ++in_seg; }
          xs.advance();
          os.advance();
        }
      }
    }
  } else if (warp >= kQpEpi0) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpi));
    // ===================== epilogue: one thread per weight row and token half =====================
    const int quad = warp & 3, half = (warp - kQpEpi0) >> 2;
    const int row = quad * 32 + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + half * kHalf;
    const uint32_t empty0 = lead(&ctl->acc_empty[0]);
    const int nseg = (steps + p.seg_steps - 1) / p.seg_steps;
    uint8_t* meta = x_ring + kQpXStages * kQpXBytes + (warp - kQpEpi0) * 64 * 8;
    pdl_wait_prior();               // y may still be read upstream
    PipeState as(kAccs);
    // down projection: slots and routing weights of a tile's rows; one trip to L2 behind the other, they took 1600 of 10300 cycles
    // at the start of each tile of 128 rows, so they are asked for during the tile before
    constexpr bool kAhead = MODE == QP_DOWN && NT == kQpTokens;     // (with few rows a tile's end does not last: 34.2 against 35.0 us)
    constexpr int kQ = MODE == QP_DOWN ? kHalf / 32 : 1;
    int slot[kQ];
    float weight[kQ];
    auto ask_slots = [&](int t) {
      const QpTile pt = qp_tile<MODE>(p, t);
#pragma unroll
      for (int q = 0; q < kQ; ++q) {
        const int r = half * kHalf + 32 * q + lane;
        slot[q] = r < pt.rows ? ld_upstream(p.order + pt.m0 + r) : -1;
      }
    };
    auto ask_weights = [&]() {
#pragma unroll
      for (int q = 0; q < kQ; ++q) weight[q] = slot[q] >= 0 ? __half2float(p.row_weights[slot[q]]) : 0.f;
    };
    if (kAhead && pair < tiles) {
      ask_slots(pair);
      ask_weights();
    }
    for (int t = pair; t < tiles; t += pairs) {
      const QpTile pt = qp_tile<MODE>(p, t);
      if (MODE == QP_DOWN) {
        if (!kAhead) {
          ask_slots(t);
          ask_weights();
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kQ; ++q) {
          reinterpret_cast<float*>(meta)[32 * q + lane] = weight[q];
          reinterpret_cast<int*>(meta + 256)[32 * q + lane] = slot[q];
        }
        __syncwarp();
        if (kAhead && t + pairs < tiles) ask_slots(t + pairs);
      }
      const int n_tile = pt.n * 2 + (int)rank;
      // weight row of this thread, and for the gate / up rows the output that the pair (lane, lane + 16) forms
      const int out = pt.n * kBlockW + (int)rank * (kBlockW / 2) + quad * 16 + (lane & 15);
      const int n = MODE == QP_GATE_UP ? out + (lane >> 4) * (p.N / 2) : n_tile * kBlockW + row;
      const bool n_ok = MODE == QP_GATE_UP ? out < p.N / 2 : n < p.N;
      // scale of group g: packed int4 tables are [tile][group][128], 8-bit tables strided by scale block
      const float* sp = p.scales;
      if (QK == Q_INT4) sp += ((int64_t)(n_ok ? n_tile : 0) * p.groups) * kBlockW + row;
      else sp += (int64_t)pt.expert * p.s_stride_e + (int64_t)((n_ok ? n : 0) / p.group_n) * p.s_stride_n;
      uint64_t acc[kHalf / 2];
#pragma unroll
      for (int j = 0; j < kHalf / 2; ++j) acc[j] = 0ull;
      if (S > 1) sp += (int64_t)(step0 / p.seg_steps) * p.s_stride_k;
      float sc = __ldg(sp);
      for (int g = 0; g < nseg; ++g) {
        const uint64_t s2 = pack_f32x2(sc, sc);
        if (g + 1 < nseg) sc = __ldg(sp + (int64_t)(g + 1) * p.s_stride_k);
        mbar_wait(&ctl->acc_full[as.stage], as.phase);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < kHalf; c += (CHAIN ? kHalf : 32)) {
          uint32_t v[CHAIN ? kHalf : 32];
          tmem_ld_32x32b_x32(taddr + as.stage * NT + c, *reinterpret_cast<uint32_t(*)[32]>(v));
          if (CHAIN && kHalf == 64) tmem_ld_32x32b_x32(taddr + as.stage * NT + c + 32, *reinterpret_cast<uint32_t(*)[32]>(v + (CHAIN ? kHalf - 32 : 0)));
          tc_wait_ld();
          if (CHAIN || c + 32 == kHalf) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(empty0 + as.stage * 8);     // in registers: the segment's buffer may be refilled
          }
#pragma unroll
          for (int j = 0; j < (CHAIN ? kHalf / 2 : 16); ++j)
            acc[c / 2 + j] = fma_f32x2(s2, pack_f32x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), acc[c / 2 + j]);
        }
        as.advance();
      }
      // ---- the tile's results ----
      if (kAhead && t + pairs < tiles) ask_weights();
      float bv = 0.f;
      if (n_ok && p.bias) bv = p.bias_is_f32 ? reinterpret_cast<const float*>(p.bias)[n]
                                             : __half2float(reinterpret_cast<const __half*>(p.bias)[n]);
      const int m0 = pt.m0 + half * kHalf;
      const int rows = pt.rows - half * kHalf;
      if (S == 1 && rows <= 0) continue;                     // uniform over the warp
      __half* y = reinterpret_cast<__half*>(p.y);
      if constexpr (S > 1) {
        // The pairs' sums meet in shared memory (over the rings: the last segment's products have read them), [token / 4][row][4], and
        // each pair adds up every S-th four tokens of its rows, in order of k.
        uint8_t* sums = w_ring + (size_t)row * 16;
#pragma unroll
        for (int j = 0; j < kHalf / 2; j += 2) {
          float f[4];
          unpack_f32x2(acc[j], f[0], f[1]);
          unpack_f32x2(acc[j + 1], f[2], f[3]);
          *reinterpret_cast<float4*>(sums + (size_t)(half * (kHalf / 4) + j / 2) * (kBlockW * 16)) = make_float4(f[0], f[1], f[2], f[3]);
        }
        __syncwarp();
        pair_sync();
        const int left = pt.rows < NT ? pt.rows : NT;
#pragma unroll 2
        for (int q = (int)(first / 2) + S * half; 4 * q < left; q += 2 * S) {
          uint4 part[S];
#pragma unroll
          for (int u = 0; u < S; ++u) part[u] = ld_cluster_128(cluster_addr(sums + (size_t)q * (kBlockW * 16), 2u * u + rank));
          float f[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int u = 0; u < S; ++u) {
            f[0] += __uint_as_float(part[u].x);
            f[1] += __uint_as_float(part[u].y);
            f[2] += __uint_as_float(part[u].z);
            f[3] += __uint_as_float(part[u].w);
          }
          const int m = pt.m0 + 4 * q;
          if (EPI == 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (n_ok && 4 * q + e < left) y[(int64_t)(m + e) * p.ldy + n] = __float2half_rn(f[e] + bv);
          } else {
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const float o = swiglu_h2(exchange_pair<1>(pack2<__half>(f[e] + bv, f[e + 1] + bv), lane));
              if (n_ok && 4 * q + e + (lane & 1) < left) y[(int64_t)(m + e + (lane & 1)) * p.ldy + (n >> 1)] = __float2half_rn(o);
            }
          }
        }
        continue;
      }
      constexpr bool kFewRows = NT < kQpTokens;              // an early end costs the large tiles 5 % (registers)
      if (MODE == QP_GATE_UP) {
        // like store_swiglu, with the pair 16 lanes apart and no further exchange (92.8 against 94.1 us for 64 experts of 190 rows)
        const bool high = lane >> 4;
        __half* yp = y + (int64_t)(m0 + (high ? 1 : 0)) * p.ldy + out;
#pragma unroll
        for (int j = 0; j < kHalf / 2; ++j) {
          if (kFewRows && 2 * j >= rows) break;
          float a, b;
          unpack_f32x2(acc[j], a, b);
          const float o = swiglu_h2(exchange_pair<16>(pack2<__half>(a, b), lane));
          if (n_ok && 2 * j + (high ? 1 : 0) < rows) *yp = __float2half_rn(o);
          yp += 2 * p.ldy;
        }
      } else if (MODE == QP_DOWN) {
        // rows go back to their slots, times the routing weight in fp32 before the rounding (fused_moe.py:201-205); in stores of
        // four outputs: 64 experts of 190 rows 84 us, of one 95
        const int col = n_tile * kBlockW + quad * 32 + (lane & ~3);
#pragma unroll
        for (int j = 0; j < kHalf / 2; j += 2) {
          if (kFewRows && 2 * j >= rows) break;
          const float4 w = *reinterpret_cast<const float4*>(meta + 8 * j);
          float f[4];
          unpack_f32x2(acc[j], f[0], f[1]);
          unpack_f32x2(acc[j + 1], f[2], f[3]);
          const uint2 v = exchange4(pack2<__half>(f[0] * w.x, f[1] * w.y), pack2<__half>(f[2] * w.z, f[3] * w.w), lane);
          const int r = 2 * j + (lane & 3);
          if (r < rows) store4(y + (int64_t)reinterpret_cast<const int*>(meta + 256)[r] * p.ldy + col, v, p.N - col, p.vec);
        }
      } else if (EPI == 0) {
        // (stores of two bytes: with few tiles per pair the exchanges of store_rows cost more than they save, 256 x 4096 x
        // 4096 int8 14.6 against 15.4 us)
        __half* yp = y + (int64_t)m0 * p.ldy + n;
        if (n_ok) {
#pragma unroll
          for (int j = 0; j < kHalf / 2; ++j) {
            float a, b;
            unpack_f32x2(acc[j], a, b);
            if (2 * j < rows) yp[0] = __float2half_rn(a + bv);
            if (2 * j + 1 < rows) yp[p.ldy] = __float2half_rn(b + bv);
            yp += 2 * p.ldy;
          }
        }
      } else {
        store_swiglu<kHalf / 2>(acc, y, p.ldy, m0, rows, (n_tile * kBlockW + quad * 32) >> 1, p.N >> 1, bv, lane, p.vec);
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsConv));
    // ===================== conversion: one thread per weight row, the two groups take alternate operand stages ==========
    // Step i of the CTA's running count belongs to group i & 1, so every op_empty barrier is waited on by one group
    // that has seen all of its phases.
    const int group = warp >> 2, quad = warp & 3;
    const int row = quad * 32 + lane, rx = row & 7;
    const uint32_t dst0 = tmem_base + ((uint32_t)(quad * 32) << 16) + kOpCol0;
    constexpr int kOwn = kOpSteps / 2;                      // operand steps of this group: group, group + 2, ...
    const uint32_t full0 = lead(&ctl->op_full[0]);
    int own = 0;
    uint32_t own_phase = 0;
    int i0 = 0;                                             // running stage count at the tile's first step
    int raw0 = 0;                                           // running raw-block count
    const int raws = (steps + kStepsPerRaw - 1) / kStepsPerRaw;
    for (int t = pair; t < tiles; t += pairs) {
      const float* zp = nullptr;
      int k = (group - i0) & 1;                             // first step of this tile that is this group's
      float z = 0.f;
      if (QK == Q_INT4) {
        const int n_tile = qp_tile<MODE>(p, t).n * 2 + (int)rank;
        zp = p.zeros + ((int64_t)(n_tile * kBlockW < p.N ? n_tile : 0) * p.groups) * kBlockW + row;
        if (k < steps) z = __ldg(zp + (int64_t)((step0 + k) / p.seg_steps) * p.s_stride_k);
      }
      for (; k < steps; k += 2) {
        __half2 add_lo, add_hi;
        if (QK == Q_INT4) {
          add_lo = __float2half2_rn(-1024.f - z);
          add_hi = __float2half2_rn(-64.f - z);
          if (k + 2 < steps) z = __ldg(zp + (int64_t)((step0 + k + 2) / p.seg_steps) * p.s_stride_k);
        }
        const int raw = raw0 + (QK == Q_INT4 ? k >> 1 : k);
        const int rs = raw % kQpWStages;
        mbar_wait(&ctl->w_full[rs], (raw / kQpWStages) & 1);
        const uint8_t* src = w_ring + (size_t)rs * kABytes + row * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          constexpr int kChunks = QK == Q_INT4 ? 2 : 4;     // 16-byte chunks of the row per 64 k
          const int stage = kSub * (group + 2 * own) + (kSub == 1 ? 0 : h);
          const int c0 = (QK == Q_INT4 ? (k & 1) * 4 : 0) + h * kChunks;
          if (CHAIN && h == 0) {
            mbar_wait(&ctl->op_empty[stage], own_phase ^ 1);
            tc_fence_after();
          }
          uint4 w[kChunks];
#pragma unroll
          for (int c = 0; c < kChunks; ++c) w[c] = lds_128(src + (((c0 + c) ^ rx) << 4));
          constexpr int kParts = CHAIN ? 1 : 2;             // 64 or 32 k at a time: 32 or 16 columns
#pragma unroll
          for (int q = 0; q < kParts; ++q) {
            uint32_t vals[32 / kParts];
#pragma unroll
            for (int c = 0; c < kChunks / kParts; ++c) {
              const uint4 v = w[q * (kChunks / kParts) + c];
              const uint32_t ws[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (QK == Q_INT4) dequant_int4_packed(ws[j], add_lo, add_hi, vals + (QK == Q_INT4 ? 16 * c + 4 * j : 0));
                else dequant_w8_word(ws[j], QK == Q_FP8, vals + (QK == Q_INT4 ? 0 : 8 * c + 2 * j));
              }
            }
            if (!CHAIN && q == 0 && (h == 0 || kSub == 2)) {
              mbar_wait(&ctl->op_empty[stage], own_phase ^ 1);
              tc_fence_after();
            }
            const uint32_t dst = dst0 + (group + 2 * own) * 64 + h * 32 + q * 16;
            if constexpr (CHAIN) tmem_st_32x32b_x32(dst, vals);
            else tmem_st_32x32b_x16(dst, vals);
          }
          if (kSub == 1 && h == 0) continue;
          if (h == 1) {
            // the raw words have all been converted: the block may be refilled (an odd last step speaks for both halves)
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(&ctl->w_empty[rs]);
              if (QK == Q_INT4 && k + 1 == steps && (k & 1) == 0) mbar_arrive(&ctl->w_empty[rs]);
            }
          }
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(full0 + stage * 8);   // barriers are 8 bytes apart
        }
        if (++own == kOwn) { own = 0; own_phase ^= 1; }
      }
      i0 += steps;
      raw0 += raws;
    }
  }

  if (S > 1 && (warp < kQpEpi0 || warp >= kQpWProd)) {
    __syncwarp();
    pair_sync();                    // the epilogue's: sums in place
  }
  tc_fence_before();
  pair_sync();                      // the peer's MMAs, commits and arrivals are over, its sums have been read
  if (warp == kQpMma) tmem_dealloc_pair(tmem_base, 512);
}

template <int QK, int EPI, int MODE, int NT, bool CHAIN, int S = 1>
static int launch_qp_form(const CUtensorMap& tw, const CUtensorMap& tx, const QuantPairParams& p, int grid, cudaStream_t st) {
  auto kern = gemm_quant_pair_kernel<QK, EPI, MODE, NT, CHAIN, S>;
  static int configured[64] = {0};
  B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, kQpSmem, configured));
  b2l_launch(kern, dim3((unsigned)grid), dim3(kQpThreads), (size_t)kQpSmem, st, tw, tx, p);
  B2L_LAUNCH_CHECK();
  return B2L_OK;
}

template <int QK, int EPI, int MODE = QP_PLAIN, int NT = kQpTokens>
static int launch_qp(const CUtensorMap& tw, const CUtensorMap& tx, const QuantPairParams& p, int grid, cudaStream_t st) {
  return p.seg_steps == 1 ? launch_qp_form<QK, EPI, MODE, NT, false>(tw, tx, p, grid, st)
                          : launch_qp_form<QK, EPI, MODE, NT, true>(tw, tx, p, grid, st);
}

template <int QK, int EPI, int S>
static int launch_qp_split(const CUtensorMap& tw, const CUtensorMap& tx, const QuantPairParams& p, cudaStream_t st) {
  const int grid = p.m_tiles * p.n_tiles * 2 * S;
  return p.seg_steps == 1 ? launch_qp_form<QK, EPI, QP_PLAIN, kQpTokens, false, S>(tw, tx, p, grid, st)
                          : launch_qp_form<QK, EPI, QP_PLAIN, kQpTokens, true, S>(tw, tx, p, grid, st);
}

// Pairs that share a tile, and the steps of each: whole raw blocks and scale groups.  A pair takes ~870 cycles a step however few of
// the SMs have a tile, so few tiles are shared by as many pairs as a whole B200 holds at once: 15 clusters of eight CTAs, 22 of six, 33
// of four.  Set-up, exchange and the larger cluster cost ~3 us, and what else would run decides from which k on they pay (us, else ->
// shared, int4 in groups of 128 / fp8 in blocks / int8 per row):
//   * grouped scales where the streaming kernel shares k as well (up to half the SMs have a tile), and one scale per row with too few
//     tiles for the plain pair form: from 8 steps on.  2048 x 1024 at 128 tokens 8.8 / 8.4 / 10.5 -> 6.7 / 6.5 / 6.5, 896 x 4864 at 256
//     13.8 / 14.0 / 17.7 -> 10.0 / 9.4 / 9.6, 4096 x 14336 at 128 (three pairs a tile) 46 / 40 / 45 -> 23 / 21 / 22
//   * where that is one wave without shares: from 18 steps on with three pairs (5632 x 2048 at 128 tokens, 16 steps: 10.1 / 9.8 / 9.3
//     -> 10.0 / 9.7 / 9.8; 5376 x 2304, 18 steps: 10.8 / 10.4 / 10.0 -> 9.9 / 9.7 / 9.8), from 24 with two (2048 x 2048 at 384: 10.0 /
//     9.8 / 9.3 -> 10.2 / 10.0 / 10.0; 4096 x 3072 at 256, 24 steps: 13.5 / 13.4 / 12.7 -> 13.0 / 12.3 / 12.4; 4096 x 14336 at 256:
//     66 / 59 / 45 -> 32 / 30 / 30)
//   * a single weight tile leaves half of each pair to padding, and then two pairs are too few against the streaming kernel's parts
//     (2821 x 128 x 8192, 23 tiles: 17.7 / 17.7 against 21.4 / 19.1).
// The same for the form with the activation, whose result is the plain form's to the bit (5632 x 2048 at 65 tokens 13.6 -> 9.1).  Sums
// in order of k, in fp32; error against 64 bits of seven shapes as before, up to 0.05 % smaller per row (shorter accumulations).
static int qp_splits(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k, int64_t* part) {
  const int64_t tiles = cdiv64(M, kQpTokens) * cdiv64(N, 2 * kBlockW), steps = cdiv64(K, kQpStepK), sms = b2l_num_sms();
  if (M <= 64 || sms < 132) return 1;
  const bool one_part = group_k >= K ? tiles >= 16 : cdiv64(M, 64) * cdiv64(N, kBlockW) > sms / 2;
  int64_t unit = group_k >= K ? 1 : group_k / kQpStepK;
  if (qk == Q_INT4 && unit % 2 != 0) unit *= 2;
  for (int s = 4; s > 1; --s) {
    if (tiles > (s == 4 ? 15 : s == 3 ? 22 : 33) || steps < (!one_part ? 8 : s == 2 ? 24 : 18)) continue;
    if (s == 2 && !one_part && N <= kBlockW) continue;
    *part = cdiv64(cdiv64(steps, s), unit) * unit;
    if ((s - 1) * *part < steps) return s;
  }
  return 1;
}

// Where the pair kernel is the faster one: with shared tiles as above, else (both kernels measured over 72 - 512 tokens, eight
// projection shapes, int4 with and without the activation and fp8 in blocks) as soon as the streaming kernel's 128 x 64 tiles need a second wave.  int4, us,
// streaming -> pair: one wave, 6144 x 4096 at 128 tokens 17 / 21, 4096 x 14336 at 72 45 / 64 (at 256, 66 / 64); two, 6144 x
// 4096 at 256 33 -> 21, 9728 x 896 at 192 (two waves of pair tiles as well) 13.8 -> 10.8; five against four, 28672 x 4096 at 192
// 94 -> 75; at 4096 tokens 1853 -> 900.
// One segment over all of k (a scale per output row) leaves the streaming kernel a single MMA warp; there the pair
// kernel wins as soon as it has 16 tiles (int8, 896 x 4864, 512 tokens 27 -> 19; 320 tokens, 12 tiles: level).
// Up to 64 tokens (tiles of 64, six conversion stages) the batch kernel is asked first and faster (gemm_quant_batch.cu).  What
// it leaves: 49 - 64 tokens with more weight tiles than SMs (28672 x 4096, int8: 26 here, 28 there), which are more than 40 tiles
// of this kernel, and callers without its workspace, which this kernel does not need.  For those, against the streaming kernel
// (int8, 32 tokens): 28672 x 4096 82 -> 28, 4096 x 4096 16.1 -> 14.5, but 4096 x 14336 (long k, 16 tiles) 37 / 45.
bool quant_pair_wanted(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k) {
  // segments of whole operand stages, or one segment over all of K
  if (group_k % kQpStepK != 0 && group_k < K) return false;
  if (qk == Q_INT4 && K % kQpStepK != 0) return false;      // the packed tables are read per 128 k
  const int64_t sms = b2l_num_sms();
  const int64_t tiles = cdiv64(M, kQpTokens) * cdiv64(N, 2 * kBlockW);
  int64_t part;
  if (qp_splits(qk, M, N, K, group_k, &part) > 1) return true;
  if (group_k >= K) return M > 64 ? tiles >= 16 : qk != Q_INT4 && (tiles >= 40 || (tiles >= 16 && K <= 4096));
  if (M <= 64) return false;
  return cdiv64(M, 64) * cdiv64(N, kBlockW) > sms;
}

// Operand stages that one accumulation in tensor memory may run over where one scale covers all of k.  A longer chain is
// further from the exact sum (4096 x 14336, 65 - 128 tokens: an error 0.23 % larger over all of k than in two parts, most of
// both being the rounding to fp16).  Where the streaming kernel would split k to fill the SMs the chain ends where its parts
// do, and the epilogue adds up the segments in fp32; with more tiles than SMs there is no split and no drain before the end.
static int qp_chain_steps(int64_t M, int64_t N, int64_t K) {
  const int64_t tiles = cdiv64(N, kBlockW) * cdiv64(M, 64), sms = b2l_num_sms(), steps = cdiv64(K, kQpStepK);
  int64_t parts = tiles < sms ? sms / tiles : 1;
  if (parts > steps / 4) parts = steps / 4 > 0 ? steps / 4 : 1;
  return (int)cdiv64(steps, parts);
}

// steps of 128 k that one scale covers, or one accumulation where a scale covers all of k
static int qp_seg_steps(int64_t M, int64_t N, int64_t K, int64_t group_k) {
  return group_k >= K ? qp_chain_steps(M, N, K) : (int)(group_k / kQpStepK);
}

int quant_pair_form(int qk, int64_t M, int64_t N, int64_t K, int64_t group_k, int swiglu) {
  if (!quant_pair_wanted(qk, M, N, K, group_k)) return 0;
  if (quant_wide_wanted(qk, M, N, cdiv64(K, kQpStepK), qp_seg_steps(M, N, K, group_k), swiglu)) return -1;
  int64_t part;
  return qp_splits(qk, M, N, K, group_k, &part);
}

int quant_pair_gemm(int qk, QuantPairParams& p, const void* x, int64_t ldx, const void* w, int64_t w_stride_bytes,
                    int64_t M, int64_t N, int64_t K, int64_t group_k, int swiglu, cudaStream_t st) {
  const int pairs = b2l_num_sms() / 2;
  p.M = (int)M; p.N = (int)N;
  p.steps = (int)cdiv64(K, kQpStepK);
  p.groups = group_k >= K ? 1 : (int)(K / group_k);
  if (qk == Q_INT4) p.s_stride_k = kBlockW;
  p.seg_steps = qp_seg_steps(M, N, K, group_k);
  if (group_k >= K) p.s_stride_k = 0;
  p.vec = p.ldy % 4 == 0 && (uintptr_t)p.y % 8 == 0;
  p.m_tiles = (int)cdiv64(M, kQpTokens);
  p.n_tiles = (int)cdiv64(N, 2 * kBlockW);
  const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles;
  const int grid = 2 * (int)(tiles < pairs ? tiles : pairs);
  CUtensorMap tw, tx;
  int rc;
  if (qk == Q_INT4) rc = b2l_make_tmap_2d(&tw, w, TMA_I32, (uint64_t)N, (uint64_t)(K / 8), (uint64_t)w_stride_bytes, kBlockW, 32, true);
  else rc = b2l_make_tmap_2d(&tw, w, TMA_U8, (uint64_t)N, (uint64_t)K, (uint64_t)w_stride_bytes, kBlockW, 128, true);
  if (rc != B2L_OK) return rc;
  rc = b2l_make_tmap_2d(&tx, x, TMA_F16, (uint64_t)M, (uint64_t)K, (uint64_t)ldx * 2, kQpTokens / 2, 64, true);
  if (rc != B2L_OK) return rc;
  if (quant_wide_wanted(qk, M, N, p.steps, p.seg_steps, swiglu)) return quant_wide_gemm(qk, p, tw, tx, swiglu, st);
  int64_t part = 0;
  const int splits = qp_splits(qk, M, N, K, group_k, &part);
  p.split_steps = (int)part;
#define QP_SPLIT(QK, EPI)                                      \
  (splits == 4 ? launch_qp_split<QK, EPI, 4>(tw, tx, p, st)    \
               : splits == 3 ? launch_qp_split<QK, EPI, 3>(tw, tx, p, st) : launch_qp_split<QK, EPI, 2>(tw, tx, p, st))
  if (splits > 1) {
    if (qk == Q_INT4) return swiglu ? QP_SPLIT(Q_INT4, 1) : QP_SPLIT(Q_INT4, 0);
    return qk == Q_FP8 ? QP_SPLIT(Q_FP8, 0) : QP_SPLIT(Q_INT8, 0);
  }
#undef QP_SPLIT
  if (qk == Q_INT4) return swiglu ? launch_qp<Q_INT4, 1>(tw, tx, p, grid, st) : launch_qp<Q_INT4, 0>(tw, tx, p, grid, st);
  if (M <= 64)
    return qk == Q_FP8 ? launch_qp<Q_FP8, 0, QP_PLAIN, 64>(tw, tx, p, grid, st) : launch_qp<Q_INT8, 0, QP_PLAIN, 64>(tw, tx, p, grid, st);
  if (qk == Q_FP8) return launch_qp<Q_FP8, 0>(tw, tx, p, grid, st);
  return launch_qp<Q_INT8, 0>(tw, tx, p, grid, st);
}

// Row boxes of the tensor map of W in the grouped modes: 16 (gate | up interleaved) or a CTA's 128 rows.
template <int MODE>
static int grouped(int qk, const MoePairGemm& g, cudaStream_t st) {
  const int pairs = b2l_num_sms() / 2;
  QuantPairParams p;
  p.y = g.y; p.ldy = g.ldy; p.bias = nullptr; p.bias_is_f32 = 0;
  p.scales = g.scales; p.s_stride_e = g.s_stride_e; p.s_stride_n = g.s_stride_n; p.s_stride_k = g.s_stride_k;
  p.zeros = nullptr;
  p.group_n = (int)(g.group_n > g.N ? g.N : g.group_n);
  p.table = g.table; p.order = g.order; p.row_weights = (const __half*)g.row_weights;
  p.M = (int)g.rows; p.N = (int)g.N;
  p.steps = (int)cdiv64(g.K, kQpStepK);
  p.groups = 0;
  p.seg_steps = g.group_k >= g.K ? p.steps : (int)(g.group_k / kQpStepK);
  p.vec = p.ldy % 4 == 0 && (uintptr_t)p.y % 8 == 0;
  p.m_tiles = 0;
  p.n_tiles = (int)cdiv64(g.N, 2 * kBlockW);
  const int64_t most = (int64_t)g.max_tiles * p.n_tiles;
  const int grid = 2 * (int)(most < pairs ? most : pairs);
  CUtensorMap tw, tx;
  int rc = b2l_make_tmap_2d(&tw, g.w, TMA_U8, (uint64_t)g.experts * g.N, (uint64_t)g.K, (uint64_t)g.w_row_stride,
                            MODE == QP_GATE_UP ? 16 : kBlockW, 128, true);
  if (rc != B2L_OK) return rc;
  rc = b2l_make_tmap_2d(&tx, g.x, TMA_F16, (uint64_t)g.rows, (uint64_t)g.K, (uint64_t)g.ldx * 2, 16, 64, true);
  if (rc != B2L_OK) return rc;
  if (g.tile_rows == 64) return qk == Q_FP8 ? launch_qp<Q_FP8, 0, MODE, 64>(tw, tx, p, grid, st) : launch_qp<Q_INT8, 0, MODE, 64>(tw, tx, p, grid, st);
  return qk == Q_FP8 ? launch_qp<Q_FP8, 0, MODE>(tw, tx, p, grid, st) : launch_qp<Q_INT8, 0, MODE>(tw, tx, p, grid, st);
}
static int moe_pair_gate_up(int qk, const MoePairGemm& g, cudaStream_t st) { return grouped<QP_GATE_UP>(qk, g, st); }
static int moe_pair_down(int qk, const MoePairGemm& g, cudaStream_t st) { return grouped<QP_DOWN>(qk, g, st); }

}  // namespace gemm

// The products of a routed layer with 8-bit experts over rows sorted by expert; `table` and `order` are b2l_moe_sort's with
// the same tile_rows.  gate_up: y[r, i] = silu(gate_i) * up_i for the sorted row r, w [E, n, k] with the gate rows first;
// down: y[slot, :] = topk_weights[slot] * (x[r] . w), slot = order[r].
extern "C" int b2l_moe_pair_gemm(void* y, const void* x, const void* w, int weight_is_fp8, const void* scales,
                                 const void* topk_weights, const void* order, const void* table, int64_t max_tiles,
                                 int tile_rows, int64_t rows, int num_experts, int64_t n, int64_t k, int64_t x_row_stride,
                                 int64_t w_row_stride, int64_t y_row_stride, int64_t group_n, int64_t group_k,
                                 int64_t s_stride_e, int64_t s_stride_n, int64_t s_stride_k, int down, void* stream) {
  using namespace gemm;
  B2L_REQUIRE(y && x && w && scales && table && (!down || (topk_weights && order)), "moe_pair_gemm: null pointer");
  B2L_REQUIRE(num_experts >= 1 && n > 0 && k > 0 && rows >= 0 && max_tiles >= 0 && (int64_t)num_experts * n < (1ll << 31),
              "moe_pair_gemm: bad shape");
  B2L_REQUIRE(k % 16 == 0 && x_row_stride % 8 == 0 && w_row_stride % 16 == 0, "moe_pair_gemm: rows must be 16-byte multiples");
  B2L_REQUIRE(group_n >= 1 && group_k >= 1 && (group_k >= k || group_k % kQpStepK == 0),
              "moe_pair_gemm: group_k (%lld) must be a multiple of %d unless it covers K", (long long)group_k, kQpStepK);
  B2L_REQUIRE(tile_rows == 64 || tile_rows == 128, "moe_pair_gemm: tile_rows %d (64 or 128)", tile_rows);
  B2L_REQUIRE(down || n % 2 == 0, "moe_pair_gemm: gate|up needs an even number of rows");
  if (rows == 0 || max_tiles == 0) return B2L_OK;
  MoePairGemm g;
  g.y = y; g.ldy = y_row_stride; g.x = x; g.ldx = x_row_stride; g.w = w; g.w_row_stride = w_row_stride;
  g.scales = (const float*)scales; g.s_stride_e = s_stride_e; g.s_stride_n = s_stride_n; g.s_stride_k = s_stride_k;
  g.group_n = group_n; g.group_k = group_k; g.experts = num_experts; g.rows = rows; g.N = n; g.K = k;
  g.table = (const int32_t*)table; g.max_tiles = max_tiles; g.tile_rows = tile_rows; g.order = (const int32_t*)order; g.row_weights = topk_weights;
  const int qk = weight_is_fp8 ? Q_FP8 : Q_INT8;
  return down ? moe_pair_down(qk, g, (cudaStream_t)stream) : moe_pair_gate_up(qk, g, (cudaStream_t)stream);
}
