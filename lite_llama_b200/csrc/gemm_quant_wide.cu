// Weight-only quantised GEMMs of large prompt batches on CTA pairs, 256 weight rows x 256 tokens per tile (entries:
// gemm_quant.cu; the kernel of 128 tokens per tile, its numerics and its layouts: gemm_quant_pair.cu).
//
// Bound: the tensor pipe and the power cap once the weights are converted half as often; what stood in the way was the trip
// of an accumulator.  One scale group is 128 k: 512 cycles of MMAs per 128 tokens, after which commit, wake-up, the loads of
// the epilogue warps, their arrival and the issuer's turn take about 1000 more (clock stamps), so that two accumulators of 128
// tokens left the pipe idle for a third of the time, and a single issuing warp, whose waits and 8 MMAs take 870 cycles for 128
// tokens, was the bottleneck before that.  Here
//   * a pair of SMs takes 256 tokens as two halves: the converted operand is used twice, so one group of four conversion warps
//     is enough, and the epilogue's threads hold both halves' sums (128 per thread);
//   * three accumulators of 128 tokens take turns over the (segment, half) units; the operand keeps 128 columns, handed over
//     and back in stages of 64 k;
//   * two warps issue, one per half;
//   * at the end of a tile lanes exchange values for stores of four outputs: 64 or 32 bytes of a token per store kept the
//     accumulators waiting for 9000 cycles of a 33000-cycle tile (4096 k, with the activation);
//   * tiles of a last wave that leaves half of the pairs idle or more are cut in two.
// The roles' registers decide: with 48 registers for the issuers 28672 x 4096 at 2048 tokens, int4, takes 502 us instead of 402
// (with 72, 20 - 40 bytes of spills are left in all roles together).
// Measured, us, 128 tokens per tile -> this kernel, launches in a row: 28672 x 4096 with the activation, int4, 4000 tokens 1198
// -> 815 (1.15 PFLOP/s), 2048 tokens 578 -> 409; 4096 x 14336, 2048 tokens, int4 291 -> 215, int8 with one scale per row 242 -> 194.
// The same bits.  (With two issuers of its own the kernel of 128 tokens per tile takes 494 and 236 us for the second and the third of
// these, and stays the faster one for a short k and for 8-bit weights in groups of 128: quant_wide_wanted.)  Int4, 2048 x 28672 x 4096:
// the tensor pipe active 64 % of the cycles, with one scale per row 92 % (profiles/pairs_and_shares_ncu.txt).
#define B2L_HANG_NORETURN true   // common.cuh: 128 accumulators beside the wait loops
#include "gemm_tc.cuh"
#include "gemm_quant_pair.cuh"
#include "pair.cuh"
#include "dequant.cuh"
#include "gemm_quant_out.cuh"

namespace gemm {

namespace {

constexpr int kQwThreads = 16 * 32;
constexpr int kQwWStages = 4, kQwXStages = 9, kQwAcc = 3;
constexpr int kQwOpStages = 4;                              // of 64 k: a step's halves of k are converted and handed back one by one
constexpr int kQwHalf = 128;                                // tokens per accumulator; each CTA stages half of them
constexpr int kQwStepK = 128;                               // k per step
constexpr int kQwXSub = kQwHalf / 2 * kStageKBytes;         // 64 tokens x 64 k
constexpr int kQwXBytes = 2 * kQwXSub;
constexpr int kQwSmem = 1024 + 1024 + kQwWStages * kABytes + kQwXStages * kQwXBytes;
constexpr int kQwBand = 8;
constexpr int kQwEpi0 = 4, kQwWProd = 12, kQwXProd = 13, kQwMma = 14;   // four conversion, eight epilogue warps
constexpr int kQwOpCol0 = kQwAcc * kQwHalf;

struct __align__(8) QwControl {
  uint64_t w_full[kQwWStages];      // own: a raw weight block has landed
  uint64_t w_empty[kQwWStages];     // own: its words have been converted (4 warp arrivals per operand stage in it)
  uint64_t x_full[kQwXStages];      // leader: both CTAs' parts of 128 tokens have landed
  uint64_t x_empty[kQwXStages];     // both: the MMAs that read them have retired
  uint64_t op_full[kQwOpStages];    // leader: both CTAs' converted rows are in tensor memory (8 warp arrivals)
  uint64_t op_empty[kQwOpStages];   // both: the MMAs of both halves have retired (two commits)
  uint64_t acc_full[kQwAcc];        // both: a segment of 128 tokens is complete
  uint64_t acc_empty[kQwAcc];       // leader: both CTAs' epilogue warps have read it (16 warp arrivals)
  uint32_t tmem_base;
};
static_assert(sizeof(QwControl) <= 1024, "control block too large");
static_assert(kQwSmem <= 227 * 1024, "shared memory");

// The tiles from `split_from` on, those of a last wave that would leave half of the pairs idle or more, are cut in two.
struct QwTile { int n, m0, rows, halves; };
__device__ __forceinline__ QwTile qw_tile(const QuantPairParams& p, int t) {
  int part = -1;
  if (t >= p.split_from) {
    part = (t - p.split_from) & 1;
    t = p.split_from + ((t - p.split_from) >> 1);
  }
  const PairTile pt = pair_tile(t, p.m_tiles, p.n_tiles, kQwBand);
  QwTile o;
  o.n = pt.n;
  o.m0 = pt.m * 2 * kQwHalf + (part > 0 ? kQwHalf : 0);
  o.rows = p.M - o.m0;                                      // of both halves and beyond; none: nothing to do
  o.halves = o.rows <= 0 ? 0 : part >= 0 || o.rows <= kQwHalf ? 1 : 2;
  return o;
}
// tokens of a half rounded up to what cta_group::2 takes as N
__device__ __forceinline__ int qw_half_n(int rows_left) {
  const int n = (rows_left + 31) & ~31;
  return n < kQwHalf ? n : kQwHalf;
}

template <int QK, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kQwThreads, 1)
gemm_quant_wide_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                       const QuantPairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  QwControl* ctl = reinterpret_cast<QwControl*>(smem);
  uint8_t* w_ring = smem + 1024;
  uint8_t* x_ring = w_ring + kQwWStages * kABytes;
  constexpr int kStepsPerRaw = QK == Q_INT4 ? 2 : 1;       // a raw block is 128 rows x 128 bytes

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = pair_rank();
  const int pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
  const int tiles = p.tiles;
  const int steps = p.steps;                               // of 128 k per tile
  if (threadIdx.x == kQwWProd * 32) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_x);
    for (int s = 0; s < kQwWStages; ++s) {
      mbar_init(&ctl->w_full[s], 1);
      mbar_init(&ctl->w_empty[s], 4 * kStepsPerRaw);
    }
    for (int s = 0; s < kQwXStages; ++s) {
      mbar_init(&ctl->x_full[s], 1);
      mbar_init(&ctl->x_empty[s], 1);
    }
    for (int s = 0; s < kQwOpStages; ++s) {
      mbar_init(&ctl->op_full[s], 8);
      mbar_init(&ctl->op_empty[s], 2);
    }
    for (int s = 0; s < kQwAcc; ++s) {
      mbar_init(&ctl->acc_full[s], 1);
      mbar_init(&ctl->acc_empty[s], 16);
    }
    mbar_fence_init();
  }
  if (warp == kQwMma) {
    tmem_alloc_pair(&ctl->tmem_base, 512);
    tmem_relinquish_pair();
    pdl_launch_dependents();        // after the allocation (gemm_dense.cu)
  }
  tc_fence_before();
  pair_sync();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  // registers per lane: four warpgroups x 128 at launch = 72 + 2 x 184 + 72
  if (warp >= kQwWProd) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    if (warp == kQwWProd) {
      // ===================== raw weight blocks of this CTA's 128 rows =====================
      PipeState ws(kQwWStages);
      const int raws = (steps + kStepsPerRaw - 1) / kStepsPerRaw;
      for (int t = pair; t < tiles; t += pairs) {
        const QwTile pt = qw_tile(p, t);
        if (pt.halves == 0) continue;
        const int row = pt.n * 2 * kBlockW + (int)rank * kBlockW;
        for (int rb = 0; rb < raws; ++rb) {
          mbar_wait(&ctl->w_empty[ws.stage], ws.phase ^ 1);
          if (elect_one()) {
            mbar_arrive_expect_tx(&ctl->w_full[ws.stage], kABytes);
            tma_load_2d_hint(w_ring + (size_t)ws.stage * kABytes, &tmap_w, rb * (QK == Q_INT4 ? 32 : 128), row,
                             &ctl->w_full[ws.stage], kEvictNormal);
          }
          __syncwarp();
          ws.advance();
        }
      }
    } else if (warp == kQwXProd) {
      // ===================== activations: this CTA's part of each half's tokens =====================
      pdl_wait_prior();
      PipeState xs(kQwXStages);
      for (int t = pair; t < tiles; t += pairs) {
        const QwTile pt = qw_tile(p, t);
        for (int s = 0; s < steps; ++s) {
          for (int h = 0; h < pt.halves; ++h) {
            const int row = pt.m0 + h * kQwHalf + (int)rank * (qw_half_n(pt.rows - h * kQwHalf) / 2);
            mbar_wait(&ctl->x_empty[xs.stage], xs.phase ^ 1);
            if (elect_one()) {
              uint8_t* dst = x_ring + (size_t)xs.stage * kQwXBytes;
              const uint32_t bar = leader_addr(&ctl->x_full[xs.stage]);
              if (rank == 0) mbar_arrive_expect_tx(&ctl->x_full[xs.stage], 2 * kQwXBytes);
              tma_load_2d_pair(dst, &tmap_x, s * kQwStepK, row, bar, kEvictNormal);
              tma_load_2d_pair(dst + kQwXSub, &tmap_x, s * kQwStepK + 64, row, bar, kEvictNormal);
            }
            __syncwarp();
            xs.advance();
          }
        }
      }
      // every stage handed back: no commit is still on its way to this CTA's barriers when it leaves
      for (int s = 0; s < kQwXStages; ++s) {
        mbar_wait(&ctl->x_empty[xs.stage], xs.phase ^ 1);
        xs.advance();
      }
    } else if (rank == 0) {
      // ===================== MMA issuers (leader), one per half =====================
      // A tile of one half is the first one's alone; the other one waits for its end, so that neither waits for a barrier that
      // is two phases behind.  A slot of X may have been the other half's: its last use is kQwXStages items back, at least four steps
      // (more behind tiles of one half).  The operand stage, waited for first, was handed back two steps ago by both issuers, so both
      // are past that use, and the slot's barrier is at most one phase behind.
      static_assert((kQwXStages - 1) / 2 >= kQwOpStages / 2, "a slot of X is used again after the operand stages have gone round");
      const uint64_t x_desc0 = umma_desc_sw128_kmajor(smem_u32(x_ring));
      PipeState xs(kQwXStages), os(kQwOpStages), as(kQwAcc);
      const int h = warp - kQwMma;
      if (h != 0) as.advance();                            // accumulator of this issuer's next unit (segment and half)
      for (int t = pair; t < tiles; t += pairs) {
        const QwTile pt = qw_tile(p, t);
        if (pt.halves == 0) continue;
        const bool both = pt.halves == 2, mine = h == 0 || both;
        const uint32_t idesc = umma_idesc(1u, 0u, 0u, 0u, 0u, 2 * kBlockW, (uint32_t)qw_half_n(pt.rows - h * kQwHalf));
        int in_seg = 0;
        for (int s = 0; s < steps; ++s) {
          const bool last = in_seg + 1 == p.seg_steps || s + 1 == steps;
          if (mine) {
            int x_stage = xs.stage + h;
            uint32_t x_phase = xs.phase;
            if (x_stage == kQwXStages) { x_stage = 0; x_phase ^= 1; }
            const uint32_t acc = tmem_base + as.stage * kQwHalf, a = tmem_base + kQwOpCol0 + os.stage * 32;
            const uint64_t b = x_desc0 + (uint64_t)((x_stage * kQwXBytes) >> 4);
            mbar_wait(&ctl->op_full[os.stage], os.phase);
            mbar_wait(&ctl->x_full[x_stage], x_phase);
            if (in_seg == 0) mbar_wait(&ctl->acc_empty[as.stage], as.phase ^ 1);
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_pair_ts(acc, a + 8 * k, b + (uint64_t)(2 * k), idesc, (in_seg | k) != 0 ? 1u : 0u);
              tc_commit_pair(&ctl->op_empty[os.stage]);
              if (!both) tc_commit_pair(&ctl->op_empty[os.stage]);
            }
            __syncwarp();
            mbar_wait(&ctl->op_full[os.stage + 1], os.phase);
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_pair_ts(acc, a + 32 + 8 * k, b + (uint64_t)((kQwXSub >> 4) + 2 * k), idesc, 1u);
              if (last) tc_commit_pair(&ctl->acc_full[as.stage]);
              tc_commit_pair(&ctl->op_empty[os.stage + 1]);
              if (!both) tc_commit_pair(&ctl->op_empty[os.stage + 1]);
              tc_commit_pair(&ctl->x_empty[x_stage]);   // the last one: the X producers wait for it before they leave
            }
            __syncwarp();
          }
          xs.advance();
          if (both) xs.advance();
          if (last) {
            as.advance();
            if (both) as.advance();
            in_seg = 0;
          } else {
            ++in_seg;
          }
          os.advance();
          os.advance();
        }
        if (!both) asm volatile("bar.sync 1, 64;" ::: "memory");
      }
    }
  } else if (warp >= kQwEpi0) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    // ===================== epilogue: one thread per weight row and 64 tokens of each half =====================
    const int quad = warp & 3, part = (warp - kQwEpi0) >> 2;
    const int row = quad * 32 + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + part * 64;
    const uint32_t empty0 = leader_addr(&ctl->acc_empty[0]);
    const int nseg = (steps + p.seg_steps - 1) / p.seg_steps;
    pdl_wait_prior();               // y may still be read upstream
    PipeState as(kQwAcc);
    for (int t = pair; t < tiles; t += pairs) {
      const QwTile pt = qw_tile(p, t);
      if (pt.halves == 0) continue;
      const int n_tile = pt.n * 2 + (int)rank;
      const int n = n_tile * kBlockW + row;
      const bool n_ok = n < p.N;
      // scale of group g: packed int4 tables are [tile][group][128], 8-bit tables strided by scale block
      const float* sp = p.scales;
      if (QK == Q_INT4) sp += ((int64_t)(n_ok ? n_tile : 0) * p.groups) * kBlockW + row;
      else sp += (int64_t)((n_ok ? n : 0) / p.group_n) * p.s_stride_n;
      uint64_t acc[2][32];
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[0][j] = acc[1][j] = 0ull;
      float sc = __ldg(sp);
      for (int g = 0; g < nseg; ++g) {
        const uint64_t s2 = pack_f32x2(sc, sc);
        if (g + 1 < nseg) sc = __ldg(sp + (int64_t)(g + 1) * p.s_stride_k);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (h < pt.halves) {
            mbar_wait(&ctl->acc_full[as.stage], as.phase);
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              uint32_t v[32];
              tmem_ld_32x32b_x32(taddr + as.stage * kQwHalf + c * 32, v);
              tc_wait_ld();
              if (c == 1) {
                // in registers: the segment's buffer may be refilled
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(empty0 + as.stage * 8);
              }
#pragma unroll
              for (int j = 0; j < 16; ++j)
                acc[h][c * 16 + j] = fma_f32x2(s2, pack_f32x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])),
                                               acc[h][c * 16 + j]);
            }
            as.advance();
          }
        }
      }
      // ---- the tile's results: lanes exchange values until each has four neighbouring outputs of one token ----
      float bv = 0.f;
      if (n_ok && p.bias) bv = p.bias_is_f32 ? reinterpret_cast<const float*>(p.bias)[n]
                                             : __half2float(reinterpret_cast<const __half*>(p.bias)[n]);
      __half* y = reinterpret_cast<__half*>(p.y);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int m0 = pt.m0 + h * kQwHalf + part * 64;
        const int rows = h < pt.halves ? pt.rows - h * kQwHalf - part * 64 : 0;
        if (rows <= 0) continue;
        if (EPI == 0) store_rows<32>(acc[h], y, p.ldy, m0, rows, n_tile * kBlockW + quad * 32, p.N, bv, lane, p.vec);
        else store_swiglu<32>(acc[h], y, p.ldy, m0, rows, (n_tile * kBlockW + quad * 32) >> 1, p.N >> 1, bv, lane, p.vec);
      }
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
    // ===================== conversion: one thread per weight row =====================
    const int row = warp * 32 + lane, rx = row & 7;
    const uint32_t dst0 = tmem_base + ((uint32_t)(warp * 32) << 16) + kQwOpCol0;
    const uint32_t full0 = leader_addr(&ctl->op_full[0]);
    PipeState os(kQwOpStages), ws(kQwWStages);
    for (int t = pair; t < tiles; t += pairs) {
      const QwTile pt = qw_tile(p, t);
      if (pt.halves == 0) continue;
      const float* zp = nullptr;
      float z = 0.f;
      if (QK == Q_INT4) {
        const int n_tile = pt.n * 2 + (int)rank;
        zp = p.zeros + ((int64_t)(n_tile * kBlockW < p.N ? n_tile : 0) * p.groups) * kBlockW + row;
        z = __ldg(zp);
      }
      int in_seg = 0;
      for (int k = 0; k < steps; ++k) {
        __half2 add_lo, add_hi;
        if (QK == Q_INT4) {
          add_lo = __float2half2_rn(-1024.f - z);
          add_hi = __float2half2_rn(-64.f - z);
          if (++in_seg == p.seg_steps) {
            in_seg = 0;
            zp += p.s_stride_k;
            if (k + 1 < steps) z = __ldg(zp);
          }
        }
        if (QK != Q_INT4 || (k & 1) == 0) mbar_wait(&ctl->w_full[ws.stage], ws.phase);
        const uint8_t* src = w_ring + (size_t)ws.stage * kABytes + row * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          constexpr int kChunks = QK == Q_INT4 ? 2 : 4;     // 16-byte chunks of the row per 64 k
          const int c0 = (QK == Q_INT4 ? (k & 1) * 4 : 0) + h * kChunks;
          uint4 w[kChunks];
#pragma unroll
          for (int c = 0; c < kChunks; ++c) w[c] = lds_128(src + (((c0 + c) ^ rx) << 4));
#pragma unroll
          for (int q = 0; q < 2; ++q) {                     // 32 k at a time: 16 columns
            uint32_t vals[16];
#pragma unroll
            for (int c = 0; c < kChunks / 2; ++c) {
              const uint4 v = w[q * (kChunks / 2) + c];
              const uint32_t ws4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (QK == Q_INT4) dequant_int4_packed(ws4[j], add_lo, add_hi, vals + (QK == Q_INT4 ? 4 * j : 0));
                else dequant_w8_word(ws4[j], QK == Q_FP8, vals + (QK == Q_INT4 ? 0 : 8 * c + 2 * j));
              }
            }
            if (q == 0) {
              mbar_wait(&ctl->op_empty[os.stage], os.phase ^ 1);
              tc_fence_after();
            }
            tmem_st_32x32b_x16(dst0 + os.stage * 32 + q * 16, vals);
          }
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(full0 + os.stage * 8);   // barriers are 8 bytes apart
          os.advance();
        }
        // the raw words have all been converted: the block may be refilled (an odd last step speaks for both halves)
        if (lane == 0) {
          mbar_arrive(&ctl->w_empty[ws.stage]);
          if (QK == Q_INT4 && k + 1 == steps && (k & 1) == 0) mbar_arrive(&ctl->w_empty[ws.stage]);
        }
        if (QK != Q_INT4 || (k & 1) == 1 || k + 1 == steps) ws.advance();
      }
    }
  }

  tc_fence_before();
  pair_sync();                      // the peer's MMAs, commits and arrivals are over
  if (warp == kQwMma) tmem_dealloc_pair(tmem_base, 512);
}

template <int QK, int EPI>
int launch_qw(const CUtensorMap& tw, const CUtensorMap& tx, const QuantPairParams& p, int grid, cudaStream_t st) {
  auto kern = gemm_quant_wide_kernel<QK, EPI>;
  static int configured[64] = {0};
  B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, kQwSmem, configured));
  b2l_launch(kern, dim3((unsigned)grid), dim3(kQwThreads), (size_t)kQwSmem, st, tw, tx, p);
  B2L_LAUNCH_CHECK();
  return B2L_OK;
}

}  // namespace

// Tiles of a last wave that leaves half of the pairs idle or more are cut in two.
static bool qw_split(int64_t tiles, int64_t pairs) { return tiles % pairs * 2 <= pairs; }

// Where it is the faster one.  Both kernels' times are waves x (steps of 128 k x time per step + set-up and end of a tile) + start, with
// a wave of tiles cut in two beside full ones; the ends of a wide tile take longer and nothing covers them, so a short k keeps the tiles
// of 128 tokens.  The ratios below (hundredths of a step of the kernel of 128 tokens) are fitted to both kernels over 81 - 366 sizes of
// 129 - 8192 tokens per kind; the choice is within 3 % of the faster one but in 3 of 285, 1 of 81 and 12 of 366.  us, 128 tokens per tile /
// this: int4 in groups of 128, 1024 x 9728 x 896 31.4 / 34.5, 1664 x 4096 x 14336 (a wave and a cut one) 181 / 198, 1024 x 4096 x 14336
// 112 / 102, 4096 x 28672 x 4096 937 / 841; one scale per row, int8, 1024 x 9728 x 896 20.7 / 22.2, 2048 x 28672 x 4096 459 / 353.  8-bit weights
// in groups of 128, whose two issuers leave it nothing to gain, stay there (fp8 in blocks, 2048 x 28672 x 4096 435 / 468, 1664 x 4096 x
// 14336 167 / 209).  With the activation the end of a tile is the heavier one in both: by waves alone (1024 x 9728 x 896 29.3 / 27.6, 2048 x
// 28672 x 4096 494 / 427; within 3 % of the faster in 128 of 128).
bool quant_wide_wanted(int qk, int64_t M, int64_t N, int64_t steps, int64_t seg_steps, int swiglu) {
  if (M <= kQwHalf || (qk != Q_INT4 && seg_steps == 1)) return false;
  const int64_t pairs = b2l_num_sms() / 2, n_tiles = cdiv64(N, 2 * kBlockW);
  const int64_t wide = cdiv64(M, 2 * kQwHalf) * n_tiles, waves = cdiv64(cdiv64(M, kQwHalf) * n_tiles, pairs);
  const bool cut = wide % pairs != 0 && qw_split(wide, pairs);
  const int64_t full = cut ? wide / pairs : cdiv64(wide, pairs);
  if (waves < 2) return false;
  if (swiglu && seg_steps == 1) return full * 150 + (cut ? 127 : 0) < 100 * waves;
  struct Cost { int step, tile, cut_step, cut_tile, start, narrow_tile, narrow_start; };
  constexpr Cost kGroups{173, 240, 141, -17, 1221, 39, 953}, kLong{143, 381, 134, -195, 2109, 12, 1688}, kRow8{153, 5, 140, -273, 2810, -59, 1939};
  const Cost c = qk != Q_INT4 ? kRow8 : seg_steps == 1 ? kGroups : kLong;
  const int64_t narrow = waves * (100 * steps + c.narrow_tile) + c.narrow_start;
  return full * (c.step * steps + c.tile) + (cut ? c.cut_step * steps + c.cut_tile : 0) + c.start < narrow * (qk != Q_INT4 ? 98 : 100) / 100;
}

// p: filled by quant_pair_gemm but for the tiles
int quant_wide_gemm(int qk, QuantPairParams& p, const CUtensorMap& tw, const CUtensorMap& tx, int swiglu, cudaStream_t st) {
  const int pairs = b2l_num_sms() / 2;
  p.m_tiles = (int)cdiv64(p.M, 2 * kQwHalf);
  const int tiles = p.m_tiles * p.n_tiles;
  p.split_from = qw_split(tiles, pairs) ? tiles - tiles % pairs : tiles;
  p.tiles = tiles + (tiles - p.split_from);
  const int grid = 2 * (p.tiles < pairs ? p.tiles : pairs);
  if (qk == Q_INT4) return swiglu ? launch_qw<Q_INT4, 1>(tw, tx, p, grid, st) : launch_qw<Q_INT4, 0>(tw, tx, p, grid, st);
  return qk == Q_FP8 ? launch_qw<Q_FP8, 0>(tw, tx, p, grid, st) : launch_qw<Q_INT8, 0>(tw, tx, p, grid, st);
}

}  // namespace gemm
