// Dense projections of prompt-sized batches on CTA pairs: Y[m, n] = sum_k X[m, k] W[n, k], fp16 / bf16 (F.linear,
// lite_llama/models/quantization/methods/unquantized.py:21-22) or int8 x int8 (lite_llama/kernels/quantization/
// w8a8.py:75-130).
//
// Bound: the tensor pipe.  What the one-SM kernel (gemm_dense.cu, 128 weight rows x 256 tokens per CTA, one tile per
// CTA) lost at these sizes: the accumulator was drained with the tensor pipe idle, every output element was a 2-byte
// store, and a CTA fetched 48 KiB per 64 k of its 128 x 256 tile.  Here
//   * a pair of SMs owns a 256-token x BN-output tile (cta_group::2): 32 KiB per SM and 64 k for twice the FLOPs;
//   * the grid is persistent and the accumulator double buffered in tensor memory (2 x BN columns), so a tile is
//     written out under the next tile's MMAs;
//   * tokens are the MMA rows, so a thread holds consecutive outputs of one token: 16-byte shared-memory writes and
//     one TMA store per warp and 64 outputs, clipped at the edges by the TMA unit.
// Measured, launches by themselves (bf16, 4096 x 28672 x 4096): 974 us (988 TFLOP/s) -> 582 us (1652 TFLOP/s); int8 768 us ->
// 289 us (3.3 POP/s); the tensor pipe is busy for 94 % of the active cycles (1024 tokens, profiles/pair_gemm_ncu.txt).  In a pass
// that keeps the card at its power cap they take 15 - 20 % longer: a feed-forward of 4096 tokens, 4096 x 14336, is 1200 us
// where its launches by themselves add up to 1030.
#include "gemm_tc.cuh"
#include "gemm_pair.cuh"
#include "pair.cuh"
#include <type_traits>

namespace gemm {

constexpr int kPairThreads = 6 * 32;          // TMA producer, MMA issuer, four epilogue warps
constexpr int kPairStages = 6;
constexpr int kPairRows = 128;                // tokens per CTA (256 per pair)
constexpr int kPairStageBytes = 2 * 128 * kStageKBytes;   // 128 token rows + up to 128 weight rows x 128 bytes of K
constexpr int kPairOut = 4 * 2 * 32 * 128;    // per epilogue warp two 32-row x 128-byte output boxes
constexpr int kPairSmem = 1024 + 1024 + kPairStages * kPairStageBytes + kPairOut;
constexpr int kPairBand = 16;                 // token tiles per band: 16 x 256 rows x 4096 x 2 bytes = 32 MiB of L2

struct PairParams {
  const void* bias;
  const float* a_scale;
  const float* b_scale;
  int M, N, num_kb, m_tiles, n_tiles;
  int vec;                          // int8: scales and bias are 16-byte aligned
};

struct __align__(8) PairControl {
  uint64_t full[kPairStages];       // leader: both CTAs' operands of a stage have landed
  uint64_t empty[kPairStages];      // both: the MMAs of a stage have retired
  uint64_t acc_full[2];             // both: a tile's accumulator is complete
  uint64_t acc_empty[2];            // leader: all eight epilogue warps have read it
  uint32_t tmem_base;
};
static_assert(sizeof(PairControl) <= 1024, "control block too large");

// 64 consecutive values from index n0, zeros from N on (N and n0 are multiples of 8): the same address in every lane
__device__ __forceinline__ void load_row64(float* dst, const float* src, int n0, int N, int vec) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int n = n0 + 8 * j;
    if (vec) {
#pragma unroll
      for (int q = 0; q < 8; q += 4) {
        const float4 f = n < N ? __ldg(reinterpret_cast<const float4*>(src + n + q)) : make_float4(0.f, 0.f, 0.f, 0.f);
        dst[8 * j + q] = f.x; dst[8 * j + q + 1] = f.y; dst[8 * j + q + 2] = f.z; dst[8 * j + q + 3] = f.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) dst[8 * j + q] = n < N ? __ldg(src + n + q) : 0.f;
    }
  }
}

template <int KIND, typename T, int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                 const __grid_constant__ CUtensorMap tmap_y, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  PairControl* ctl = reinterpret_cast<PairControl*>(smem);
  uint8_t* ring = smem + 1024;
  uint8_t* out_stage = ring + kPairStages * kPairStageBytes;
  constexpr int kXBytes = kPairRows * kStageKBytes, kWBytes = BN / 2 * kStageKBytes;
  constexpr int kKPerStage = KIND == 0 ? 64 : 128;
  constexpr int kTmemCols = 512;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = pair_rank();
  const int pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
  const int tiles = p.m_tiles * p.n_tiles;
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_y);
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&ctl->acc_full[b], 1);
      mbar_init(&ctl->acc_empty[b], 8);
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&ctl->tmem_base, kTmemCols);
    tmem_relinquish_pair();
    pdl_launch_dependents();        // after the allocation (gemm_dense.cu)
  }
  tc_fence_before();
  pair_sync();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  if (warp == 0) {
    // ===================== TMA producer: this CTA's halves of both operands =====================
    pdl_wait_prior();
    PipeState ps(kPairStages);
    for (int t = pair; t < tiles; t += pairs) {
      const PairTile pt = pair_tile(t, p.m_tiles, p.n_tiles, kPairBand);
      const int row_x = pt.m * 2 * kPairRows + (int)rank * kPairRows;
      const int row_w = pt.n * BN + (int)rank * (BN / 2);
      for (int kb = 0; kb < p.num_kb; ++kb) {
        mbar_wait(&ctl->empty[ps.stage], ps.phase ^ 1);
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(&ctl->full[ps.stage], 2 * (kXBytes + kWBytes));
          uint8_t* st = ring + (size_t)ps.stage * kPairStageBytes;
          const uint32_t bar = leader_addr(&ctl->full[ps.stage]);
          tma_load_2d_pair(st, &tmap_x, kb * kKPerStage, row_x, bar, kEvictNormal);
          tma_load_2d_pair(st + kXBytes, &tmap_w, kb * kKPerStage, row_w, bar, kEvictNormal);
        }
        __syncwarp();
        ps.advance();
      }
    }
    // every stage handed back: no commit is still on its way to this CTA's barriers when it leaves
    for (int s = 0; s < kPairStages; ++s) {
      mbar_wait(&ctl->empty[ps.stage], ps.phase ^ 1);
      ps.advance();
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (leader only) =====================
    if (rank == 0) {
      constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      constexpr uint32_t idesc = KIND == 0 ? umma_idesc(1u, fmt, fmt, 0u, 0u, 2 * kPairRows, BN)
                                           : umma_idesc(2u, 1u, 1u, 0u, 0u, 2 * kPairRows, BN);
      const uint64_t desc0 = umma_desc_sw128_kmajor(smem_u32(ring));
      PipeState ps(kPairStages);
      int it = 0;
      for (int t = pair; t < tiles; t += pairs, ++it) {
        const int buf = it & 1;
        mbar_wait(&ctl->acc_empty[buf], ((it >> 1) & 1) ^ 1);
        tc_fence_after();
        for (int kb = 0; kb < p.num_kb; ++kb) {
          mbar_wait(&ctl->full[ps.stage], ps.phase);
          tc_fence_after();
          if (elect_one()) {
            const uint64_t xd = desc0 + (uint64_t)((ps.stage * kPairStageBytes) >> 4);
            const uint64_t wd = xd + (uint64_t)(kXBytes >> 4);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_pair<KIND>(tmem_base + buf * 256, xd + 2 * k, wd + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
            tc_commit_pair(&ctl->empty[ps.stage]);
            if (kb + 1 == p.num_kb) tc_commit_pair(&ctl->acc_full[buf]);
          }
          __syncwarp();
          ps.advance();
        }
      }
    }
  } else {
    // ===================== epilogue: one thread per token row =====================
    const int quad = warp & 3;
    uint8_t* mine = out_stage + (size_t)quad * 2 * 4096;
    const uint32_t empty0 = leader_addr(&ctl->acc_empty[0]), empty1 = leader_addr(&ctl->acc_empty[1]);
    const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
    pdl_wait_prior();               // activation scales are upstream data; y may still be read upstream
    int it = 0, box = 0;
    for (int t = pair; t < tiles; t += pairs, ++it) {
      const PairTile pt = pair_tile(t, p.m_tiles, p.n_tiles, kPairBand);
      const int buf = it & 1;
      const int m_warp = pt.m * 2 * kPairRows + (int)rank * kPairRows + quad * 32;
      float sa = 1.f;
      if (KIND == 1) sa = p.a_scale[m_warp + lane < p.M ? m_warp + lane : p.M - 1];
      // int8: weight scales (and bias) of 64 outputs in 16-byte loads, requested 64 outputs ahead.  One 4-byte load per output
      // behind the sums took 10 us per tile (256 x 37888 x 3584: 40.6 -> 32.0 us, x 1792 30.6 -> 18.2)
      float sb[KIND == 1 ? 64 : 1], bb[KIND == 1 ? 64 : 1];
      auto scales = [&](int n0) {
        if (KIND == 1) {
          load_row64(sb, p.b_scale, n0, p.N, p.vec);
          if (p.bias) load_row64(bb, reinterpret_cast<const float*>(p.bias), n0, p.N, p.vec);
        }
      };
      scales(pt.n * BN);
      mbar_wait(&ctl->acc_full[buf], (it >> 1) & 1);
      tc_fence_after();
#pragma unroll 1
      for (int c = 0; c < BN; c += 64) {
        uint32_t v[64];
        tmem_ld_32x32b_x32(taddr + buf * 256 + c, *reinterpret_cast<uint32_t(*)[32]>(v));
        tmem_ld_32x32b_x32(taddr + buf * 256 + c + 32, *reinterpret_cast<uint32_t(*)[32]>(v + 32));
        tc_wait_ld();
        if (c + 64 == BN) {         // the accumulator is in registers: the next tile but one may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(buf ? empty1 : empty0);
        }
        const int n0 = pt.n * BN + c;
        if (n0 >= p.N || m_warp >= p.M) continue;       // uniform over the warp
        uint8_t* dst = mine + (box & 1) * 4096;
        if (lane == 0) bulk_wait_read<1>();             // the store that used this box two boxes ago has read it
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          uint32_t o[4];
          const int n = n0 + 8 * j;
          const bool in = n < p.N;                      // N is a multiple of 8
          if (KIND == 0) {
            uint4 b4 = make_uint4(0u, 0u, 0u, 0u);
            if (p.bias && in) b4 = ldg_128(reinterpret_cast<const T*>(p.bias) + n);
            const T* b = reinterpret_cast<const T*>(&b4);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float f0 = __uint_as_float(v[8 * j + 2 * q]), f1 = __uint_as_float(v[8 * j + 2 * q + 1]);
              if (p.bias) { f0 += to_f32(b[2 * q]); f1 += to_f32(b[2 * q + 1]); }
              o[q] = pack2<T>(f0, f1);
            }
          } else {
            // acc.float * a_scale[m] * b_scale[n] (+ bias), in this order (w8a8.py:117-123)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int e = 8 * j + 2 * q;
              float f0 = (float)(int)v[e] * sa * sb[KIND == 1 ? e : 0];
              float f1 = (float)(int)v[e + 1] * sa * sb[KIND == 1 ? e + 1 : 0];
              if (p.bias) { f0 += bb[KIND == 1 ? e : 0]; f1 += bb[KIND == 1 ? e + 1 : 0]; }
              o[q] = pack2<T>(f0, f1);
            }
          }
          *reinterpret_cast<uint4*>(dst + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        if (c + 64 < BN) scales(n0 + 64);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmap_y, dst, n0, m_warp);
          bulk_commit();
        }
        ++box;
      }
    }
    if (lane == 0) bulk_wait_all();
  }

  tc_fence_before();
  pair_sync();                      // the peer's MMAs, commits and arrivals are over
  if (warp == 1) tmem_dealloc_pair(tmem_base, kTmemCols);
}

// ---------------------------------------------------------------------------------------------------------------
// Few tiles: S pairs of one cluster share a tile, each with its part of k, and add up in shared memory.
//
// Bound: with 14 to 33 tiles of 256 x 256 most SMs were idle, or (one-SM kernel) smaller tiles fetched the weights once per 64
// tokens: 256 x 3584 x 18944 moved 400 MB through L2 in 38 us.  A split of k through global memory costs a trip to L2 per
// partial tile of 128 KiB and a wait for CTAs that may not run yet; CTAs of a cluster do run together.  Each CTA leaves its 128 x
// BN sums in its own shared memory (the ring is idle by then), [BN / 4][row][4] so that 16-byte accesses of a warp are
// consecutive, and CTA s adds up columns [s BN / S, ...) of its rows over the S CTAs of its rank parity, in order of s.
// Measured: pair_splits below.
// ---------------------------------------------------------------------------------------------------------------
template <int KIND, typename T, int BN, int S>
__global__ void __cluster_dims__(2 * S, 1, 1) __launch_bounds__(kPairThreads, 1)
gemm_pair_split_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
                       const __grid_constant__ CUtensorMap tmap_y, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  PairControl* ctl = reinterpret_cast<PairControl*>(smem);
  uint8_t* ring = smem + 1024;
  uint8_t* out_stage = ring + kPairStages * kPairStageBytes;
  constexpr int kXBytes = kPairRows * kStageKBytes, kWBytes = BN / 2 * kStageKBytes;
  constexpr int kKPerStage = KIND == 0 ? 64 : 128;
  constexpr int kCols = BN / S;                 // outputs that this CTA adds up
  static_assert(kCols % 64 == 0 && kPairRows * BN * 4 <= kPairStages * kPairStageBytes, "split");

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = pair_rank(), side = rank & 1u, first = rank & ~1u;      // side 0: leader of the pair
  const int split = (int)(rank >> 1), tile = (int)blockIdx.x / (2 * S);
  const PairTile pt = pair_tile(tile, p.m_tiles, p.n_tiles, kPairBand);
  const int kb0 = (int)((int64_t)p.num_kb * split / S), kb1 = (int)((int64_t)p.num_kb * (split + 1) / S);
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_y);
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(&ctl->full[s], 1);
      mbar_init(&ctl->empty[s], 1);
    }
    mbar_init(&ctl->acc_full[0], 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&ctl->tmem_base, 256);
    tmem_relinquish_pair();
    pdl_launch_dependents();        // after the allocation (gemm_dense.cu)
  }
  tc_fence_before();
  pair_sync();
  tc_fence_after();
  const uint32_t tmem_base = ctl->tmem_base;

  if (warp == 0) {
    // ===================== TMA producer: this CTA's halves of both operands =====================
    const int row_x = pt.m * 2 * kPairRows + (int)side * kPairRows, row_w = pt.n * BN + (int)side * (BN / 2);
    auto expect = [&](int stage) {
      if (side == 0) mbar_arrive_expect_tx(&ctl->full[stage], 2 * (kXBytes + kWBytes));
    };
    auto load = [&](int stage, int kb, bool weights) {
      uint8_t* st = ring + (size_t)stage * kPairStageBytes;
      const uint32_t bar = cluster_addr(&ctl->full[stage], first);
      if (weights) tma_load_2d_pair(st + kXBytes, &tmap_w, kb * kKPerStage, row_w, bar, kEvictNormal);
      else tma_load_2d_pair(st, &tmap_x, kb * kKPerStage, row_x, bar, kEvictNormal);
    };
    // weights are static: the first stages' are requested before the previous kernel has ended
    const int pre = kb1 - kb0 < kPairStages ? kb1 - kb0 : kPairStages;
    if (elect_one())
      for (int i = 0; i < pre; ++i) { expect(i); load(i, kb0 + i, true); }
    __syncwarp();
    pdl_wait_prior();
    if (elect_one())
      for (int i = 0; i < pre; ++i) load(i, kb0 + i, false);
    __syncwarp();
    PipeState ps(kPairStages);
    for (int i = 0; i < pre; ++i) ps.advance();
    for (int kb = kb0 + pre; kb < kb1; ++kb) {
      mbar_wait(&ctl->empty[ps.stage], ps.phase ^ 1);
      if (elect_one()) {
        expect(ps.stage);
        load(ps.stage, kb, true);
        load(ps.stage, kb, false);
      }
      __syncwarp();
      ps.advance();
    }
    // every stage handed back: no commit is still on its way when the ring is overwritten
    for (int s = 0; s < pre; ++s) {
      if (pre < kPairStages) mbar_wait(&ctl->empty[s], 0);
      else { mbar_wait(&ctl->empty[ps.stage], ps.phase ^ 1); ps.advance(); }
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (leader only) =====================
    if (side == 0) {
      constexpr uint32_t fmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
      constexpr uint32_t idesc = KIND == 0 ? umma_idesc(1u, fmt, fmt, 0u, 0u, 2 * kPairRows, BN)
                                           : umma_idesc(2u, 1u, 1u, 0u, 0u, 2 * kPairRows, BN);
      const uint64_t desc0 = umma_desc_sw128_kmajor(smem_u32(ring));
      PipeState ps(kPairStages);
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(&ctl->full[ps.stage], ps.phase);
        tc_fence_after();
        if (elect_one()) {
          const uint64_t xd = desc0 + (uint64_t)((ps.stage * kPairStageBytes) >> 4);
          const uint64_t wd = xd + (uint64_t)(kXBytes >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_pair<KIND>(tmem_base, xd + 2 * k, wd + 2 * k, idesc, (kb - kb0) | k ? 1u : 0u);
          tc_commit_pair_at(&ctl->empty[ps.stage], first);
          if (kb + 1 == kb1) tc_commit_pair_at(&ctl->acc_full[0], first);
        }
        __syncwarp();
        ps.advance();
      }
    }
  } else {
    // ===================== this CTA's sums to shared memory =====================
    const int row = (warp & 3) * 32 + lane;
    const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
    mbar_wait(&ctl->acc_full[0], 0);
    tc_fence_after();
#pragma unroll 1
    for (int c = 0; c < BN; c += 64) {
      uint32_t v[64];
      tmem_ld_32x32b_x32(taddr + c, *reinterpret_cast<uint32_t(*)[32]>(v));
      tmem_ld_32x32b_x32(taddr + c + 32, *reinterpret_cast<uint32_t(*)[32]>(v + 32));
      tc_wait_ld();
#pragma unroll
      for (int j = 0; j < 16; ++j)
        *reinterpret_cast<uint4*>(ring + ((size_t)(c / 4 + j) * kPairRows + row) * 16) =
            make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
  }
  tc_fence_before();
  pair_sync();                      // all sums of the cluster are in place
  if (warp >= 2) {
    // ===================== a part of the columns over all splits =====================
    const int quad = warp & 3, row = quad * 32 + lane;
    uint8_t* mine = out_stage + (size_t)quad * 2 * 4096;
    const int m_warp = pt.m * 2 * kPairRows + (int)side * kPairRows + quad * 32;
    pdl_wait_prior();               // activation scales are upstream data; y may still be read upstream
    float sa = 1.f;
    if (KIND == 1) sa = p.a_scale[m_warp + lane < p.M ? m_warp + lane : p.M - 1];
#pragma unroll 1
    for (int c = 0; c < kCols; c += 64) {
      const int c0 = split * kCols + c, n0 = pt.n * BN + c0;
      if (n0 >= p.N || m_warp >= p.M) continue;         // uniform over the warp
      float sb[KIND == 1 ? 64 : 1], bb[KIND == 1 ? 64 : 1];
      if (KIND == 1) {
        load_row64(sb, p.b_scale, n0, p.N, p.vec);
        if (p.bias) load_row64(bb, reinterpret_cast<const float*>(p.bias), n0, p.N, p.vec);
      }
      uint8_t* dst = mine + (c / 64 & 1) * 4096;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint4 part[S][2];
#pragma unroll
        for (int s = 0; s < S; ++s) {
          const uint32_t src = cluster_addr(ring + ((size_t)(c0 / 4 + 2 * j) * kPairRows + row) * 16, 2u * s + side);
          part[s][0] = ld_cluster_128(src);
          part[s][1] = ld_cluster_128(src + kPairRows * 16);
        }
        uint32_t v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint32_t* w0 = reinterpret_cast<const uint32_t*>(&part[0][0]);
          v[q] = w0[q];
#pragma unroll
          for (int s = 1; s < S; ++s) {
            const uint32_t w = reinterpret_cast<const uint32_t*>(&part[s][0])[q];
            v[q] = KIND == 0 ? __float_as_uint(__uint_as_float(v[q]) + __uint_as_float(w)) : v[q] + w;
          }
        }
        uint32_t o[4];
        const int n = n0 + 8 * j;
        if (KIND == 0) {
          uint4 b4 = make_uint4(0u, 0u, 0u, 0u);
          if (p.bias && n < p.N) b4 = ldg_128(reinterpret_cast<const T*>(p.bias) + n);
          const T* b = reinterpret_cast<const T*>(&b4);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float f0 = __uint_as_float(v[2 * q]), f1 = __uint_as_float(v[2 * q + 1]);
            if (p.bias) { f0 += to_f32(b[2 * q]); f1 += to_f32(b[2 * q + 1]); }
            o[q] = pack2<T>(f0, f1);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int e = KIND == 1 ? 8 * j + 2 * q : 0, e1 = KIND == 1 ? e + 1 : 0;
            float f0 = (float)(int)v[2 * q] * sa * sb[e], f1 = (float)(int)v[2 * q + 1] * sa * sb[e1];
            if (p.bias) { f0 += bb[e]; f1 += bb[e1]; }
            o[q] = pack2<T>(f0, f1);
          }
        }
        *reinterpret_cast<uint4*>(dst + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmap_y, dst, n0, m_warp);
        bulk_commit();
      }
    }
    if (lane == 0) bulk_wait_all();
  }
  pair_sync();                      // the peers have read this CTA's sums
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 256);
  }
}

// Output columns per pair tile: waves x tile width is what the grid spends on the tensor pipe.  A 128-wide tile re-fetches
// the activations twice as often and reaches 1.25 PFLOP/s where the 256-wide one reaches 1.65 (bf16, 4096 tokens), so it
// has to win by that ratio: it does when the wide tiles leave most pairs idle (512 x 4096 outputs: 32 tiles for 74 pairs).
static int pair_bn(int64_t m_tiles, int64_t N, int pairs) {
  const int64_t w256 = cdiv64(m_tiles * cdiv64(N, 256), pairs) * 256;
  const int64_t w128 = cdiv64(m_tiles * cdiv64(N, 128), pairs) * 128;
  return w128 * 132 < w256 * 100 ? 128 : 256;
}

// How many pairs share a tile: four or two where all clusters are in one wave and the parts of k outweigh the sum at their end.
// us, whichever kernel had the call -> split: 4 pairs, 256 x 3584 x 18944 bf16 69 -> 33, int8 38 -> 19.5; 96 tokens (half of the
// rows are padding) 40 -> 30 and 26 -> 18.5; 192 x 1024 x 2048 11.2 -> 8.8 and 11.0 -> 7.8; 2 pairs, 256 x 4096 x 14336 53 -> 39 and
// 30 -> 24, 512 x 2048 x 4096 18 -> 16 and 13.4 -> 11.9.  Not: 192 x 3328 x 1024 bf16 7.2 / 8.9, 512 x 2048 x 768 6.9 / 8.4, 1024 x 2048 x
// 4096 int8 12.5 / 13.4 (64 tiles of 128 outputs fill the pairs), 384 x 512 x 8192 bf16 14.8 / 16.0 (four tiles: the one-SM kernel
// splits k further).  The limits in tiles stay below what a whole B200 holds at once, 15 clusters of eight CTAs and 33 of four;
// a part with fewer SMs may hold fewer, so below 132 nothing is shared.
static int pair_splits(int kind, const PairGemm& g) {
  const int64_t tiles = cdiv64(g.M, 2 * kPairRows) * cdiv64(g.N, 256), kb = cdiv64(g.K, kind == 0 ? 64 : 128);
  if (b2l_num_sms() < 132 || g.M <= kPairRows / 2) return 1;
  const bool low = g.M <= kPairRows;
  if (kind == 0 && !low && tiles <= 4 && kb >= 128) return 1;
  if (tiles <= 14 && kb >= (kind == 0 && !low ? 32 : 16)) return 4;
  if (!low && ((tiles <= 16 && kb >= 32) || (tiles <= 32 && kb >= 80))) return 2;
  return 1;
}

// Where the pair kernel is the faster one (both kernels measured over 64 - 4096 tokens and some thirty projection shapes, us,
// one-SM -> pair): 256 tokens x 6144 x 4096: 36 -> 18, 512 x 4096 x 4096: 36 -> 18, 2048 x 28672 x 4096: 495 -> 299, int8
// 256 x 37888 x 3584: 61 -> 32.  With up to 128 tokens half of each pair's rows are padding: only where four pairs share a tile.
// Few tiles leave pairs idle, but so do the one-SM kernel's: 38 tiles, 256 x 9728 x 896 20 -> 10.4, int8 15.8 -> 7.5; 19, 512 x
// 2432 x 1024 13.9 -> 7.0; 16, 256 x 2048 x 768 8.9 -> 5.6; 12, 256 x 1536 x 1024 9.0 -> 6.3.
bool pair_gemm_wanted(int kind, const PairGemm& g) {
  // TMA store: 16-byte rows of Y; everything else is the one-SM kernel's own alignment rule
  if (g.N % 8 != 0 || (g.ldy * 2) % 16 != 0 || (uintptr_t)g.y % 16 != 0 || (kind == 0 && g.bias && (uintptr_t)g.bias % 16 != 0))
    return false;
  const int pairs = b2l_num_sms() / 2;
  const int64_t m_tiles = cdiv64(g.M, 2 * kPairRows);
  if (pair_splits(kind, g) > 1) return true;
  return g.M > kPairRows && m_tiles * cdiv64(g.N, pair_bn(m_tiles, g.N, pairs)) >= 12;
}

template <int KIND, typename T, int BN, int S>
static int launch_split(const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& ty, const PairParams& p, cudaStream_t st) {
  auto kern = gemm_pair_split_kernel<KIND, T, BN, S>;
  static int configured[64] = {0};
  B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, kPairSmem, configured));
  b2l_launch(kern, dim3((unsigned)(p.m_tiles * p.n_tiles * 2 * S)), dim3(kPairThreads), (size_t)kPairSmem, st, tx, tw, ty, p);
  B2L_LAUNCH_CHECK();
  return B2L_OK;
}

template <int KIND, typename T, int BN>
static int launch_pair(const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& ty, const PairParams& p, int grid,
                       cudaStream_t st) {
  auto kern = gemm_pair_kernel<KIND, T, BN>;
  static int configured[64] = {0};
  B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, kPairSmem, configured));
  b2l_launch(kern, dim3((unsigned)grid), dim3(kPairThreads), (size_t)kPairSmem, st, tx, tw, ty, p);
  B2L_LAUNCH_CHECK();
  return B2L_OK;
}

int pair_gemm(int kind, int dtype, const PairGemm& g, cudaStream_t st) {
  const int pairs = b2l_num_sms() / 2;
  PairParams p;
  p.bias = g.bias; p.a_scale = g.a_scale; p.b_scale = g.b_scale;
  p.vec = ((uintptr_t)g.b_scale | (kind == 1 ? (uintptr_t)g.bias : 0)) % 16 == 0;
  p.M = (int)g.M; p.N = (int)g.N;
  p.m_tiles = (int)cdiv64(g.M, 2 * kPairRows);
  const int bn = pair_splits(kind, g) > 1 ? 256 : pair_bn(p.m_tiles, g.N, pairs);
  p.n_tiles = (int)cdiv64(g.N, bn);
  p.num_kb = (int)cdiv64(g.K, kind == 0 ? 64 : 128);
  const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles;
  const int grid = 2 * (int)(tiles < pairs ? tiles : pairs);
  const TmaElem out_el = dtype == B2L_F16 ? TMA_F16 : TMA_BF16;
  const TmaElem el = kind == 1 ? TMA_U8 : out_el;
  const uint64_t esz = kind == 1 ? 1 : 2;
  const uint32_t kbox = kind == 1 ? 128 : 64;
  const int splits = pair_splits(kind, g);
  CUtensorMap tx, tw, ty;
  int rc = b2l_make_tmap_2d(&tx, g.x, el, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.ldx * esz, kPairRows, kbox, true);
  if (rc != B2L_OK) return rc;
  rc = b2l_make_tmap_2d(&tw, g.w, el, (uint64_t)g.N, (uint64_t)g.K, (uint64_t)g.ldw * esz, (uint32_t)(bn / 2), kbox, true);
  if (rc != B2L_OK) return rc;
  rc = b2l_make_tmap_2d(&ty, g.y, out_el, (uint64_t)g.M, (uint64_t)g.N, (uint64_t)g.ldy * 2, 32, 64, true);
  if (rc != B2L_OK) return rc;
#define PAIR_SPLIT(KIND, T) (splits == 4 ? launch_split<KIND, T, 256, 4>(tx, tw, ty, p, st) : launch_split<KIND, T, 256, 2>(tx, tw, ty, p, st))
  if (splits > 1) {
    if (kind == 0) return dtype == B2L_F16 ? PAIR_SPLIT(0, __half) : PAIR_SPLIT(0, __nv_bfloat16);
    return dtype == B2L_F16 ? PAIR_SPLIT(1, __half) : PAIR_SPLIT(1, __nv_bfloat16);
  }
#undef PAIR_SPLIT
#define PAIR_BN(KIND, T) (bn == 128 ? launch_pair<KIND, T, 128>(tx, tw, ty, p, grid, st) : launch_pair<KIND, T, 256>(tx, tw, ty, p, grid, st))
  if (kind == 0) return dtype == B2L_F16 ? PAIR_BN(0, __half) : PAIR_BN(0, __nv_bfloat16);
  return dtype == B2L_F16 ? PAIR_BN(1, __half) : PAIR_BN(1, __nv_bfloat16);
#undef PAIR_BN
}

}  // namespace gemm
