// flash_decoding: single-token decode attention over the token-granular paged KV cache.
//
// Replaces lite_llama/kernels/flashdecoding.py:23-380 (stage-1 + stage-2 Triton kernels).
// Same contract: history of batch row b is the cache rows
//   table[b_req_idx[b], 0 .. b_seq_len[b]-1]            (flashdecoding.py:66-69)
// K/V are strided views of one [max_tokens, 2*Hkv, D] pool (models/base.py:119-123).
//
// B200 design:
//  * one CTA per (split, kv-head block, batch row) streams WHOLE TOKEN ROWS: in the fused pool a
//    token's K heads and V heads are one contiguous 2*Hkv*D*2-byte run (4 KiB for Llama-3-8B), so a
//    single 1-D bulk async copy (cp.async.bulk, the TMA engine) per token brings in
//    everything every head needs.  (First version: one CTA per kv head with 256-byte copies reached
//    only 29 % of HBM peak -- the copy engine's request rate, not bytes, was the limit.)
//  * a dedicated producer warp walks the token table and issues the copies into a 3-4 stage
//    shared-memory ring guarded by mbarriers; consumer warps never touch the LSU for K/V;
//  * one consumer warp per (kv head, block of 16 query heads): the GQA group is stacked on the M
//    dimension of the MMA tile, so each cached element is read from HBM exactly once (the reference
//    launches one program per q head and re-reads it G times);
//  * QK^T and PV on tensor cores with fp32 accumulation (fp16 products are exact in fp32, which
//    keeps the reference's "fp32 product" precision, flashdecoding.py:115-120), fp32 online softmax;
//  * split-KV sized from host-known quantities only (graph-safe); fp32 partials + log-sum-exp,
//    merged by a second small kernel (reference stage 2, flashdecoding.py:224-313); large steps: shares of the work that there
//    is, whatever rows it belongs to (flash_decode_shares_kernel);
//  * a step too small to fill the chip is bound by latency instead: its splits are the CTAs of a cluster, with as few kv
//    heads each as still fit in one wave, and merge through one another's shared memory (cluster_merge below).
#include "common.cuh"
#include <type_traits>

namespace {

constexpr int kTT = 16;            // tokens per pipeline stage (one m16n8k16 k-step of PV)
constexpr int kMaxConsumers = 8;
constexpr int kMaxStages = 4;
constexpr int kMaxCluster = 8;
constexpr int kStagesAt = 128;     // bytes of shared memory before the stages: their barriers

struct DecodeParams {
  const void* q; int64_t q_bs, q_hs;
  const void* k; int64_t k_ts, k_hs;
  const void* v; int64_t v_ts, v_hs;
  const int32_t* table; int64_t tab_bs, tab_ss;
  const void* req_idx; int req_w;
  const void* seq_len; int len_w;
  void* out; int64_t o_bs, o_hs;
  float* ws_o;    // [B, Hq, splits, D]
  float* ws_lse;  // [B, Hq, splits]   (log2 domain)
  int* tickets;   // one per (batch row, kv-head block), zero on entry and on exit; null = separate combine kernel
  int Hq, Hkv, G, qblocks;
  int HB;         // kv heads per CTA (divides Hkv)
  int copy_mode;  // 0: one copy per token (K|V fused run), 1: one K + one V copy, 2: one copy per head
  int stages;
  int chunk;      // tokens per split (multiple of kTT)
  int splits;
  float scale_log2;
};
// apart: with these the calls of the other kernels cost the host 0.36 us more (16 bytes; 8.3 -> 8.7 us a call through ctypes)
struct ShareParams : DecodeParams {
  int2* ws_info;  // first and last CTA of every (kv-head block, batch row); ws_o [head of a block, slots, D]
  int* ws_cut;    // 1: rows are cut in splits after all, ws_o [B, Hq, splits, D]
  int batch;
  int slots;      // two per CTA
};

__host__ __device__ inline int row_pitch(int HB, int D) { return 2 * HB * D * 2 + 16; }  // +16: ldmatrix conflict-free

// all threads of the cluster that have not left; what each wrote to shared memory before is visible to the others after
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_smem(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_peer(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_peer4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

// The splits of a row and head block, left by the CTAs of a cluster in their own shared memory (rows, then statistics), added up
// in split order like in the kernels below.  Every CTA takes its share of the outputs, also those whose split is empty: where
// those left before, one or two of eight CTAs made four to eight trips through shared memory for 32 heads (4 kv heads, 16 rows of
// 16 tokens under a bound of 65 8.6 us, of 20 under 80 7.4; merge kernel 5.9 and 6.9; now 5.3 and 5.4).  A way of its own for rows of
// one split took 4.0, and all others 0.2 - 0.6 longer: these steps are short enough for the size of their code to count.
template <typename T, int D>
__device__ __forceinline__ void cluster_merge(const DecodeParams& p, uint32_t part, int len) {
  const int split = blockIdx.x, heads = p.HB * p.G;
  __syncwarp();
  cluster_sync_all();
  const int nsp = (int)((unsigned)(len + p.chunk - 1) / (unsigned)p.chunk);
  for (int i = split * blockDim.x + threadIdx.x; i < heads * (D / 4); i += p.splits * blockDim.x) {
    const int local = i / (D / 4), d = i % (D / 4) * 4;
    float lse[kMaxCluster];
    float4 v[kMaxCluster];
#pragma unroll
    for (int r = 0; r < kMaxCluster; ++r)
      if (r < nsp) {
        const uint32_t peer = peer_smem(part, r);
        lse[r] = ld_peer(peer + (heads * D + local) * 4);
        v[r] = ld_peer4(peer + (local * D + d) * 4);
      }
    float M = -INFINITY, L = 0.f;
#pragma unroll
    for (int r = 0; r < kMaxCluster; ++r)
      if (r < nsp) M = fmaxf(M, lse[r]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < kMaxCluster; ++r)
      if (r < nsp) {
        const float w = fast_exp2(lse[r] - M);
        acc.x += w * v[r].x; acc.y += w * v[r].y; acc.z += w * v[r].z; acc.w += w * v[r].w;
        L += w;
      }
    uint32_t* to = reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(p.out) + (int64_t)blockIdx.z * p.o_bs +
                                               (int64_t)(blockIdx.y * heads + local) * p.o_hs + d);
    to[0] = pack2<T>(acc.x / L, acc.y / L);
    to[1] = pack2<T>(acc.z / L, acc.w / L);
  }
  __syncwarp();
  cluster_sync_all();                 // the peers have read this CTA's rows
}

// two values of which those that are not finite become 0
template <typename T>
__device__ __forceinline__ uint32_t finite2(uint32_t v) {
  typename Vec2<T>::type x = *reinterpret_cast<const typename Vec2<T>::type*>(&v), largest;
  const uint32_t most = std::is_same<T, __half>::value ? 0x7bff7bffu : 0x7f7f7f7fu;
  largest = *reinterpret_cast<const typename Vec2<T>::type*>(&most);
  return v & __hle2_mask(__habs2(x), largest);
}

// One consumer warp's work: 16 query heads (fewer: rows of zeros) of one kv head, its tiles of kTT tokens in turn.
template <typename T, int D>
struct Consumer {
  uint32_t qf[D / 16][4];             // A operand, m16 x k16 per step; rows = query heads of this KV group
  float o[D / 8][4];
  float m_run[2], l_run[2];
  bool v0, v1;                        // rows g and g + 8 exist

  __device__ __forceinline__ void begin(const DecodeParams& p, int b, int kvh, int hq0, int hq1, int tq) {
    v0 = hq0 < p.G;
    v1 = hq1 < p.G;
    const T* qb = reinterpret_cast<const T*>(p.q) + (int64_t)b * p.q_bs;
    const T* q0 = qb + (int64_t)(kvh * p.G + (v0 ? hq0 : 0)) * p.q_hs;
    const T* q1 = qb + (int64_t)(kvh * p.G + (v1 ? hq1 : 0)) * p.q_hs;
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      const int c = kk * 16 + 2 * tq;
      qf[kk][0] = v0 ? *reinterpret_cast<const uint32_t*>(q0 + c) : 0u;
      qf[kk][1] = v1 ? *reinterpret_cast<const uint32_t*>(q1 + c) : 0u;
      qf[kk][2] = v0 ? *reinterpret_cast<const uint32_t*>(q0 + c + 8) : 0u;
      qf[kk][3] = v1 ? *reinterpret_cast<const uint32_t*>(q1 + c + 8) : 0u;
    }
#pragma unroll
    for (int i = 0; i < D / 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
    m_run[0] = m_run[1] = -INFINITY;
    l_run[0] = l_run[1] = 0.f;
  }
  // the tile at shared address sb, tokens tbase .. of which those before `end` count; ka, va: ldmatrix lane addresses.
  // REST: what the probabilities lose as 16-bit operands is multiplied as well.  Of every split the largest probability is 1, which
  // loses nothing, so rows in few parts would end 2 - 5 % further from the exact result than rows in many; with it they end 19 %
  // closer.  That rest is 0 or negative for most, and 0 x inf and inf - inf are NaN, so it leaves out values that are not finite.
  template <bool REST>
  __device__ __forceinline__ void tile(const DecodeParams& p, uint32_t sb, uint32_t ka, uint32_t va, int64_t tbase, int64_t end, int tq) {
    // ---- S = Q K^T  (16 heads x 16 tokens) ----
    float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk) {
      uint32_t bf[4];
      ldmatrix_x4(bf, sb + ka + kk * 32);
      mma_m16n8k16<T>(sc[0], qf[kk], bf[0], bf[1]);
      mma_m16n8k16<T>(sc[1], qf[kk], bf[2], bf[3]);
    }
    // ---- scale, mask, online softmax (log2 domain) ----
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int64_t pos = tbase + j * 8 + 2 * tq + (e & 1);
        float v = sc[j][e] * p.scale_log2;
        v = pos < end ? v : -INFINITY;
        sc[j][e] = v;
        mx[e >> 1] = fmaxf(mx[e >> 1], v);
      }
    }
    float alpha[2], base[2];
#pragma unroll
    for (int r2 = 0; r2 < 2; ++r2) {
      mx[r2] = fmaxf(mx[r2], __shfl_xor_sync(0xffffffffu, mx[r2], 1));
      mx[r2] = fmaxf(mx[r2], __shfl_xor_sync(0xffffffffu, mx[r2], 2));
      const float mnew = fmaxf(m_run[r2], mx[r2]);
      base[r2] = mnew == -INFINITY ? 0.f : mnew;   // avoid (-inf) - (-inf)
      alpha[r2] = fast_exp2(m_run[r2] - base[r2]);
      m_run[r2] = mnew;
    }
    float ps[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float pv = fast_exp2(sc[j][e] - base[e >> 1]);
        sc[j][e] = pv;
        ps[e >> 1] += pv;
      }
    }
    l_run[0] = l_run[0] * alpha[0] + ps[0];
    l_run[1] = l_run[1] * alpha[1] + ps[1];
    // (most tiles do not raise the largest score; what REST saves here pays for the values that it leaves out: 32 kv heads of one query
    // head each, 64 rows of 250 - 500 88.4 -> 84.8 us)
    if (!REST || __any_sync(0xffffffffu, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
      for (int i = 0; i < D / 8; ++i) {
        o[i][0] *= alpha[0]; o[i][1] *= alpha[0];
        o[i][2] *= alpha[1]; o[i][3] *= alpha[1];
      }
    }
    // ---- O += P V  (P: 16 heads x 16 tokens as the A operand) ----
    uint32_t pf[4];
    pf[0] = pack2<T>(sc[0][0], sc[0][1]);
    pf[1] = pack2<T>(sc[0][2], sc[0][3]);
    pf[2] = pack2<T>(sc[1][0], sc[1][1]);
    pf[3] = pack2<T>(sc[1][2], sc[1][3]);
    uint32_t rest[4];
    if (REST) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const typename Vec2<T>::type h = *reinterpret_cast<const typename Vec2<T>::type*>(&pf[i]);
        rest[i] = pack2<T>(sc[i >> 1][2 * (i & 1)] - to_f32(h.x), sc[i >> 1][2 * (i & 1) + 1] - to_f32(h.y));
      }
    }
#pragma unroll
    for (int dn = 0; dn < D / 16; ++dn) {
      uint32_t bf[4];
      ldmatrix_x4_trans(bf, sb + va + dn * 32);
      mma_m16n8k16<T>(o[2 * dn], pf, bf[0], bf[1]);
      mma_m16n8k16<T>(o[2 * dn + 1], pf, bf[2], bf[3]);
      if (REST) {
#pragma unroll
        for (int i = 0; i < 4; ++i) bf[i] = finite2<T>(bf[i]);
        mma_m16n8k16<T>(o[2 * dn], rest, bf[0], bf[1]);
        mma_m16n8k16<T>(o[2 * dn + 1], rest, bf[2], bf[3]);
      }
    }
  }
  // quad-reduce the row sums (each lane only summed its own 4 columns per tile)
  __device__ __forceinline__ void sum_rows() {
#pragma unroll
    for (int r2 = 0; r2 < 2; ++r2) {
      l_run[r2] += __shfl_xor_sync(0xffffffffu, l_run[r2], 1);
      l_run[r2] += __shfl_xor_sync(0xffffffffu, l_run[r2], 2);
    }
  }
  // rows r2 (0: head hq0, 1: hq1) as 16-bit results or as fp32 partial rows
  __device__ __forceinline__ void store_out(const DecodeParams& p, int r2, int b, int head, float inv, int tq) const {
    T* orow = reinterpret_cast<T*>(p.out) + (int64_t)b * p.o_bs + (int64_t)head * p.o_hs;
#pragma unroll
    for (int i = 0; i < D / 8; ++i)
      *reinterpret_cast<uint32_t*>(orow + i * 8 + 2 * tq) = pack2<T>(o[i][2 * r2] * inv, o[i][2 * r2 + 1] * inv);
  }
  __device__ __forceinline__ void store_part(float* orow, int r2, float inv, int tq) const {
#pragma unroll
    for (int i = 0; i < D / 8; ++i)
      *reinterpret_cast<float2*>(orow + i * 8 + 2 * tq) = make_float2(o[i][2 * r2] * inv, o[i][2 * r2 + 1] * inv);
  }
};

// Who merges the splits of a row: a second kernel; nobody (a single split), or the last CTA (tickets); the CTAs of a cluster,
// which are the grid's x, up to kMaxCluster splits.  The second form does the first one's work as well; its code for the rest costs
// 0.2 - 0.3 us of 16 - 51, except with heads of 256, whose sums do not fit into registers and spill less in it (4 %).
enum { FD_SPLITS, FD_WHOLE, FD_CLUSTER };
// one split with tokens
template <typename T, int D, int FORM>
__device__ __forceinline__ void decode_split(const DecodeParams& p, uint8_t* smem, int64_t seq_len, int64_t start, int split, int hblk,
                                             int b, int64_t req) {
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);   // [kMaxStages]
  uint64_t* empty_bar = full_bar + kMaxStages;              // [kMaxStages]
  uint8_t* stage_base = smem + kStagesAt;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nconsumers = p.HB * p.qblocks;      // blockDim.x == (nconsumers + 1) * 32

  const int64_t end = (start + p.chunk < seq_len) ? start + p.chunk : seq_len;
  const int ntiles = (int)((end - start + kTT - 1) / kTT);

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], nconsumers);
    }
    mbar_fence_init();
  }
  __syncthreads();

  const int PITCH = row_pitch(p.HB, D);
  const int stage_bytes = kTT * PITCH;
  constexpr uint32_t HEAD_BYTES = D * 2;

  if (warp == nconsumers) {
    // ===================== producer warp: gather token rows through the table =====================
    const int32_t* trow = p.table + req * p.tab_bs;
    const int h0 = hblk * p.HB;
    const char* kbase = reinterpret_cast<const char*>(p.k) + (int64_t)h0 * p.k_hs * 2;
    const char* vbase = reinterpret_cast<const char*>(p.v) + (int64_t)h0 * p.v_hs * 2;
    const int tok = lane & 15;          // token of the tile this lane serves
    const int half = lane >> 4;         // lanes 16..31 take the V side in modes 1/2
    const uint32_t side_bytes = p.HB * HEAD_BYTES;
    int64_t pos = start + tok;
    pos = pos < end ? pos : end - 1;    // clamp: padded rows duplicate a valid row (finite data, masked later)
    int64_t row_next = trow[pos * p.tab_ss];
    int s = 0; uint32_t phase = 0;
    for (int t = 0; t < ntiles; ++t) {
      const int64_t row = row_next;
      if (t + 1 < ntiles) {
        int64_t pn = start + (int64_t)(t + 1) * kTT + tok;
        pn = pn < end ? pn : end - 1;
        row_next = trow[pn * p.tab_ss];
      }
      mbar_wait(&empty_bar[s], phase ^ 1);
      if (lane == 0) mbar_arrive_expect_tx(&full_bar[s], (uint32_t)kTT * 2u * side_bytes);
      __syncwarp();
      uint8_t* dst = stage_base + s * stage_bytes + tok * PITCH;
      if (p.copy_mode == 0) {
        if (half == 0) bulk_g2s(dst, kbase + row * p.k_ts * 2, 2u * side_bytes, &full_bar[s]);
      } else if (p.copy_mode == 1) {
        if (half == 0) bulk_g2s(dst, kbase + row * p.k_ts * 2, side_bytes, &full_bar[s]);
        else bulk_g2s(dst + side_bytes, vbase + row * p.v_ts * 2, side_bytes, &full_bar[s]);
      } else {
        const char* src = half == 0 ? kbase + row * p.k_ts * 2 : vbase + row * p.v_ts * 2;
        const int64_t hs = (half == 0 ? p.k_hs : p.v_hs) * 2;
        for (int h = 0; h < p.HB; ++h)
          bulk_g2s(dst + half * side_bytes + h * HEAD_BYTES, src + h * hs, HEAD_BYTES, &full_bar[s]);
      }
      if (++s == p.stages) { s = 0; phase ^= 1; }
    }
    if (FORM == FD_CLUSTER) __syncthreads();
  } else {
    // ===================== consumer warps: one (kv head, 16-query-head block) each =====================
    const int hl = warp / p.qblocks;            // kv head inside this CTA's block
    const int qblk = warp % p.qblocks;
    const int kvh = hblk * p.HB + hl;
    const int g = lane >> 2, tq = lane & 3;
    const int hq0 = qblk * 16 + g, hq1 = hq0 + 8;
    Consumer<T, D> c;
    c.begin(p, b, kvh, hq0, hq1, tq);

    const uint32_t k_off = hl * HEAD_BYTES;
    const uint32_t v_off = (p.HB + hl) * HEAD_BYTES;
    const int mj = lane >> 3, r8 = lane & 7;
    // ldmatrix lane addresses (relative to the stage base)
    const uint32_t ka = ((mj >> 1) * 8 + r8) * PITCH + k_off + (mj & 1) * 16;
    const uint32_t va = ((mj & 1) * 8 + r8) * PITCH + v_off + (mj >> 1) * 16;

    int s = 0; uint32_t phase = 0;
    for (int t = 0; t < ntiles; ++t) {
      mbar_wait(&full_bar[s], phase);
      const uint32_t sb = smem_u32(stage_base + s * stage_bytes);

      c.template tile<false>(p, sb, ka, va, start + (int64_t)t * kTT, end, tq);
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty_bar[s]);
      if (++s == p.stages) { s = 0; phase ^= 1; }
    }

    c.sum_rows();
    // Cluster: the partial rows go to the CTA's own shared memory, over the stages that every warp has finished with
    float* part = reinterpret_cast<float*>(stage_base);
    if (FORM == FD_CLUSTER) __syncthreads();
    // this warp saw every token of the split for its heads: write the result rows directly
#pragma unroll
    for (int r2 = 0; r2 < 2; ++r2) {
      if (!(r2 == 0 ? c.v0 : c.v1)) continue;
      const int head = kvh * p.G + (r2 == 0 ? hq0 : hq1);
      const float inv = 1.0f / c.l_run[r2];
      if (FORM == FD_CLUSTER) {
        const int local = hl * p.G + (r2 == 0 ? hq0 : hq1);
        c.store_part(part + local * D, r2, inv, tq);
        if (tq == 0) part[p.HB * p.G * D + local] = c.m_run[r2] + log2f(c.l_run[r2]);
      } else if (FORM == FD_WHOLE && p.splits == 1) {
        c.store_out(p, r2, b, head, inv, tq);
      } else {
        const int64_t off = ((int64_t)b * p.Hq + head) * p.splits + split;
        c.store_part(p.ws_o + off * D, r2, inv, tq);
        if (tq == 0) p.ws_lse[off] = c.m_run[r2] + log2f(c.l_run[r2]);
      }
    }
  }

  // ---- stage 2 folded in (reference: a second kernel, flashdecoding.py:224-313): the CTA that finishes a
  // (batch row, kv-head block) LAST merges its splits.  Deterministic: the merge always runs over all splits in index
  // order, whoever executes it.  The ticket resets itself, so graph replays start clean. ----
  if (FORM == FD_WHOLE && p.splits > 1 && p.tickets != nullptr) {
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    int nsp = (int)((seq_len + p.chunk - 1) / p.chunk);          // splits that have tokens (the others returned above)
    nsp = nsp < p.splits ? nsp : p.splits;
    if (threadIdx.x == 0) {
      int* t = p.tickets + (int64_t)b * gridDim.y + hblk;
      const int old = atomicAdd(t, 1);
      s_last = (old == nsp - 1);
      if (s_last) *t = 0;
    }
    __syncthreads();
    if (s_last) {
      __threadfence();
      const int heads_here = p.HB * p.G;
      const int head0 = hblk * p.HB * p.G;
      for (int idx = threadIdx.x; idx < heads_here * D; idx += blockDim.x) {
        const int head = head0 + idx / D, d = idx % D;
        const int64_t off = ((int64_t)b * p.Hq + head) * p.splits;
        float M = -INFINITY;
        for (int sp = 0; sp < nsp; ++sp) M = fmaxf(M, __ldcg(p.ws_lse + off + sp));
        float acc = 0.f, L = 0.f;
        for (int sp = 0; sp < nsp; ++sp) {
          const float w = fast_exp2(__ldcg(p.ws_lse + off + sp) - M);
          acc += w * __ldcg(p.ws_o + (off + sp) * D + d);
          L += w;
        }
        reinterpret_cast<T*>(p.out)[(int64_t)b * p.o_bs + (int64_t)head * p.o_hs + d] = from_f32<T>(acc / L);
      }
    }
  }
}

template <typename T, int D, int FORM>
__global__ void __launch_bounds__((kMaxConsumers + 1) * 32) flash_decode_split_kernel(const DecodeParams p) {
  pdl_prologue();   // everything below reads what earlier kernels of the step wrote (q, KV rows, lengths, table)
  extern __shared__ __align__(128) uint8_t smem[];
  const int64_t seq_len = load_index(p.seq_len, blockIdx.z, p.len_w);
  const int64_t start = (int64_t)blockIdx.x * p.chunk;
  const int most = p.chunk * kMaxCluster;                   // FD_CLUSTER: tokens that its kMaxCluster splits hold
  const int len = seq_len < most ? (int)seq_len : most;
  if (start < seq_len) {
    decode_split<T, D, FORM>(p, smem, seq_len, start, blockIdx.x, blockIdx.y, blockIdx.z, load_index(p.req_idx, blockIdx.z, p.req_w));
  } else if (FORM != FD_SPLITS && blockIdx.x == 0) {        // an empty row is zero; other empty splits have nothing to contribute
    const int heads = p.HB * p.G;
    for (int i = threadIdx.x; i < heads * (D / 2); i += blockDim.x)
      *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(p.out) + (int64_t)blockIdx.z * p.o_bs +
                                   (int64_t)(blockIdx.y * heads + i / (D / 2)) * p.o_hs + 2 * (i % (D / 2))) = 0u;
  }
  if (FORM == FD_CLUSTER && len > 0) cluster_merge<T, D>(p, smem_u32(smem + kStagesAt), len);
}

// Stage 2: log-sum-exp merge of the per-split partials (reference: flashdecoding.py:224-313).
template <typename T, int D, bool MANY>   // MANY: some row may have more than 8 splits
__global__ void flash_decode_combine_kernel(const DecodeParams p) {
  pdl_prologue();
  const int b = blockIdx.x, head = blockIdx.y;
  const int64_t seq_len = load_index(p.seq_len, b, p.len_w);
  int nsp = (int)((seq_len + p.chunk - 1) / p.chunk);
  nsp = nsp < p.splits ? nsp : p.splits;
  const int64_t off = ((int64_t)b * p.Hq + head) * p.splits;
  if (!MANY || nsp <= 8) {
    float M = -INFINITY;
    for (int s = 0; s < nsp; ++s) M = fmaxf(M, p.ws_lse[off + s]);
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
      float acc = 0.f, L = 0.f;
      for (int s = 0; s < nsp; ++s) {
        const float w = fast_exp2(p.ws_lse[off + s] - M);
        acc += w * p.ws_o[(off + s) * D + d];
        L += w;
      }
      const float val = nsp > 0 ? acc / L : 0.f;
      reinterpret_cast<T*>(p.out)[(int64_t)b * p.o_bs + (int64_t)head * p.o_hs + d] = from_f32<T>(val);
    }
    return;
  }
  // Many splits, bound by latency: the statistics of up to 32 splits are read side by side, and eight partial rows are
  // requested before the first is added; the sums run in split order (one sequence of 8000 tokens, 125 splits: 20.4 -> 16.7
  // us with the split kernel; up to 8 splits the plain loop is the faster one, 256 sequences of 300 tokens 38.6 against 41.2).
  const int lane = threadIdx.x & 31;
  float M = -INFINITY;
  for (int s = lane; s < nsp; s += 32) M = fmaxf(M, __ldcg(p.ws_lse + off + s));
  M = warp_reduce_max(M);
  for (int d0 = 0; d0 < D; d0 += blockDim.x) {          // whole warps: the weights travel by shuffles
    const int d = d0 + threadIdx.x;
    const float* src = p.ws_o + off * D + (d < D ? d : 0);
    float acc = 0.f, L = 0.f;
    for (int s0 = 0; s0 < nsp; s0 += 32) {
      const float mine = s0 + lane < nsp ? fast_exp2(__ldcg(p.ws_lse + off + s0 + lane) - M) : 0.f;
      const int n = nsp - s0 < 32 ? nsp - s0 : 32;
      for (int s1 = 0; s1 < n; s1 += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = s1 + i < n ? __ldcg(src + (int64_t)(s0 + s1 + i) * D) : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float w = __shfl_sync(0xffffffffu, mine, (s1 + i) & 31);
          if (s1 + i < n) { acc += w * v[i]; L += w; }
        }
      }
    }
    const float val = nsp > 0 ? acc / L : 0.f;
    if (d < D) reinterpret_cast<T*>(p.out)[(int64_t)b * p.o_bs + (int64_t)head * p.o_hs + d] = from_f32<T>(val);
  }
}

// Shares.  The lengths are device data, so a grid of (split, row) CTAs cut for the longest possible length spends six waves
// of short CTAs on a batch that would fill the chip once, each with the start of its ring (25 splits of 80 tokens per row, 32
// sequences of 1000 - 2000 tokens: 44 us of 30 at the rate of a copy), and larger splits lose where most rows are short.  Here every
// CTA adds up the lengths and takes its part of the work there is:
//   * no more splits with tokens than CTAs: a split each, as in the grid of splits, and with its result;
//   * else an equal share of all tiles of all rows, whatever rows they belong to: one wave, one ring that runs on from row
//     to row.  A CTA that covers a row whole writes its result; else the row's parts go to the workspace (each CTA has at most
//     two: of a row that began before it, and of one that ends after it), and the owner of a row's first tile notes its first
//     and last CTA for the merge.  A row's bits then depend on where the shares part it, hence on the other rows' lengths.
struct RowPart { int b, blk, first, last, tiles, cta_last; };   // tiles first .. last - 1 of a row of `tiles`; its last CTA

// the parts of rows that a CTA works on, in turn
struct ShareWalk {
  const int* prefix;                              // tiles of the rows before, [batch + 1]
  int batch, all, t, hi, b, blk, grid, total;
  __device__ __forceinline__ ShareWalk(const int* prefix_, int batch_, int nblk, int cta, int grid_)
      : prefix(prefix_), batch(batch_), grid(grid_) {
    all = prefix[batch];                          // of one kv-head block
    total = all * nblk;
    t = (int)((unsigned long long)cta * (unsigned)total / (unsigned)grid);
    hi = (int)((unsigned long long)(cta + 1) * (unsigned)total / (unsigned)grid);
    blk = (unsigned)t / (unsigned)all;
    b = 0;
    const int rem = t - blk * all;
    // the last row that begins at or before rem (empty rows have nothing): 32 at a time, the whole warp
    const int lane = threadIdx.x & 31;
    for (int step = batch > 32 ? 32 : 1;; step = 1) {
      const int at = b + lane * step;
      b += step * (__popc(__ballot_sync(0xffffffffu, at < batch && prefix[at] <= rem)) - 1);
      if (step == 1) break;
    }
  }
  __device__ __forceinline__ bool next(RowPart& r) {
    while (t < hi) {
      const int begin = blk * all + prefix[b], end = blk * all + prefix[b + 1], from = t - begin;
      r.b = b;
      r.blk = blk;
      if (++b == batch) { b = 0; ++blk; }
      if (end <= t) continue;                     // an empty row
      t = end < hi ? end : hi;
      r.tiles = end - begin;
      r.first = from;
      r.last = t - begin;
      r.cta_last = r.last == r.tiles ? 0 : (int)(((unsigned long long)end * (unsigned)grid - 1u) / (unsigned)total);   // 0: this one
      return true;
    }
    return false;
  }
};

// Registers of a thread: what plan_shares counts with.  Left to itself the compiler takes 168 with heads of 128, beside which fewer blocks
// of the merge kernel wait on the SM (32 kv heads, one of 1600 tokens under 8000 15.4 us instead of 12.5, four of 400 12.5 / 11.3).
__host__ __device__ constexpr int share_regs(int D) { return D == 128 ? 152 : D == 64 ? 96 : 72; }

template <typename T, int D>
__global__ void __maxnreg__(share_regs(D)) flash_decode_shares_kernel(const ShareParams p) {
  pdl_prologue();   // everything below reads what earlier kernels of the step wrote (q, KV rows, lengths, table)
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ int warp_sum[2][kMaxConsumers + 1];
  __shared__ int found[2];
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem);   // [kMaxStages]
  uint64_t* empty_bar = full_bar + kMaxStages;              // [kMaxStages]
  uint8_t* stage_base = smem + kStagesAt;
  const int PITCH = row_pitch(p.HB, D), stage_bytes = kTT * PITCH;
  constexpr uint32_t HEAD_BYTES = D * 2;
  int* prefix = reinterpret_cast<int*>(stage_base + p.stages * stage_bytes);    // [batch + 1]
  int* lens = prefix + p.batch + 1;                                             // [batch]
  int* reqs = lens + p.batch;                                                   // [batch]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nconsumers = p.HB * p.qblocks;      // blockDim.x == (nconsumers + 1) * 32
  const int nblk = p.Hkv / p.HB, grid = (int)gridDim.x, cta = blockIdx.x;

  // ---- splits with tokens; a thread owns neighbouring rows ----
  const int most = p.chunk * p.splits;          // tokens of a row that the call's bound lets count
  const int per = (p.batch + blockDim.x - 1) / blockDim.x, r_lo = threadIdx.x * per;
  const int r_hi = r_lo + per < p.batch ? r_lo + per : p.batch;
  auto units = [](int len, int tokens) { return (int)((unsigned)(len + tokens - 1) / (unsigned)tokens); };
  // of the rows before this thread's, and of all rows
  auto sum_before = [&](int own, int* sums, int& all) {
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    if (lane == 31) sums[warp] = upto;
    __syncthreads();
    const int of_warp = lane <= nconsumers ? sums[lane] : 0;
    all = __reduce_add_sync(0xffffffffu, of_warp);
    return upto - own + (int)__reduce_add_sync(0xffffffffu, lane < warp ? of_warp : 0);
  };
  int own = 0, all;
#pragma unroll 1
  for (int r = r_lo; r < r_hi; ++r) {
    const int64_t n = load_index(p.seq_len, r, p.len_w);
    reqs[r] = (int)load_index(p.req_idx, r, p.req_w);
    lens[r] = n > most ? most : n > 0 ? (int)n : 0;
    own += units(lens[r], p.chunk);
  }
  int at = sum_before(own, warp_sum[0], all);
  if (cta == 0 && threadIdx.x == 0) *p.ws_cut = nblk * all <= grid;
  if (nblk * all <= grid) {
    if (cta >= nblk * all) return;
    const int hblk = nblk == 1 ? 0 : (unsigned)cta / (unsigned)all;
    int split = cta - hblk * all - at;          // of this thread's rows
    if (split >= 0 && split < own) {
      int r = r_lo;
      for (int n; r + 1 < r_hi && split >= (n = units(lens[r], p.chunk)); ++r) split -= n;
      found[0] = r;
      found[1] = split;
    }
    __syncthreads();
    const int b = found[0];
    split = found[1];
    decode_split<T, D, FD_SPLITS>(p, smem, lens[b], (int64_t)split * p.chunk, split, hblk, b, reqs[b]);
    return;
  }

  // ---- tiles of the rows before each ----
  own = 0;
  for (int r = r_lo; r < r_hi; ++r) own += units(lens[r], kTT);
  at = sum_before(own, warp_sum[1], all);
  for (int r = r_lo; r < r_hi; ++r) {
    prefix[r] = at;
    at += units(lens[r], kTT);
  }
  if (threadIdx.x == 0) {
    prefix[p.batch] = all;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], nconsumers);
    }
    mbar_fence_init();
  }
  __syncthreads();

  ShareWalk walk(prefix, p.batch, nblk, cta, grid);
  RowPart r;
  int s = 0;
  uint32_t phase = 0;
  if (warp == nconsumers) {
    // ===================== producer warp: gather token rows through the table =====================
    const int tok = lane & 15;          // token of the tile this lane serves
    const int half = lane >> 4;         // lanes 16..31 take the V side in modes 1/2
    const uint32_t side_bytes = p.HB * HEAD_BYTES;
    // table entry of this lane's token: padded rows duplicate a valid row (finite data, masked later)
    auto entry = [&](const RowPart& at, int tile) {
      int pos = tile * kTT + tok;
      pos = pos < lens[at.b] ? pos : lens[at.b] - 1;
      return p.table[(int64_t)reqs[at.b] * p.tab_bs + (int64_t)pos * p.tab_ss];
    };
    bool more = walk.next(r);
    int tile = more ? r.first : 0;
    int64_t row_next = more ? entry(r, tile) : 0;
    while (more) {
      const int64_t row = row_next;
      const RowPart at = r;
      const bool begins = tile == 0;
      // the next tile's entry is on its way while this one waits for its stage
      if (++tile == at.last) {
        more = walk.next(r);
        tile = more ? r.first : 0;
      }
      if (more) row_next = entry(r, tile);
      const char* kbase = reinterpret_cast<const char*>(p.k) + (int64_t)at.blk * p.HB * p.k_hs * 2;
      const char* vbase = reinterpret_cast<const char*>(p.v) + (int64_t)at.blk * p.HB * p.v_hs * 2;
      mbar_wait(&empty_bar[s], phase ^ 1);
      if (lane == 0) mbar_arrive_expect_tx(&full_bar[s], (uint32_t)kTT * 2u * side_bytes);
      __syncwarp();
      uint8_t* dst = stage_base + s * stage_bytes + tok * PITCH;
      if (p.copy_mode == 0) {
        if (half == 0) bulk_g2s(dst, kbase + row * p.k_ts * 2, 2u * side_bytes, &full_bar[s]);
      } else if (p.copy_mode == 1) {
        if (half == 0) bulk_g2s(dst, kbase + row * p.k_ts * 2, side_bytes, &full_bar[s]);
        else bulk_g2s(dst + side_bytes, vbase + row * p.v_ts * 2, side_bytes, &full_bar[s]);
      } else {
        const char* src = half == 0 ? kbase + row * p.k_ts * 2 : vbase + row * p.v_ts * 2;
        const int64_t hs = (half == 0 ? p.k_hs : p.v_hs) * 2;
        for (int h = 0; h < p.HB; ++h)
          bulk_g2s(dst + half * side_bytes + h * HEAD_BYTES, src + h * hs, HEAD_BYTES, &full_bar[s]);
      }
      if (begins && lane == 0) p.ws_info[at.blk * p.batch + at.b] = make_int2(cta, at.last == at.tiles ? cta : at.cta_last);
      if (++s == p.stages) { s = 0; phase ^= 1; }
    }
  } else {
    // ===================== consumer warps: one (kv head, 16-query-head block) each =====================
    const int hl = warp / p.qblocks;            // kv head inside the block
    const int qblk = warp % p.qblocks;
    const int g = lane >> 2, tq = lane & 3;
    const int hq0 = qblk * 16 + g, hq1 = hq0 + 8;
    const uint32_t k_off = hl * HEAD_BYTES;
    const uint32_t v_off = (p.HB + hl) * HEAD_BYTES;
    const int mj = lane >> 3, r8 = lane & 7;
    // ldmatrix lane addresses (relative to the stage base)
    const uint32_t ka = ((mj >> 1) * 8 + r8) * PITCH + k_off + (mj & 1) * 16;
    const uint32_t va = ((mj & 1) * 8 + r8) * PITCH + v_off + (mj >> 1) * 16;
    Consumer<T, D> c;
    while (walk.next(r)) {
      const int kvh = r.blk * p.HB + hl;
      const int64_t end = lens[r.b];
      c.begin(p, r.b, kvh, hq0, hq1, tq);
      for (int t = r.first; t < r.last; ++t) {
        mbar_wait(&full_bar[s], phase);
        c.template tile<true>(p, smem_u32(stage_base + s * stage_bytes), ka, va, (int64_t)t * kTT, end, tq);
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[s]);
        if (++s == p.stages) { s = 0; phase ^= 1; }
      }
      c.sum_rows();
      const bool whole = r.first == 0 && r.last == r.tiles;
#pragma unroll
      for (int r2 = 0; r2 < 2; ++r2) {
        if (!(r2 == 0 ? c.v0 : c.v1)) continue;
        const int hq = r2 == 0 ? hq0 : hq1;
        const float inv = 1.0f / c.l_run[r2];
        if (whole) {
          c.store_out(p, r2, r.b, kvh * p.G + hq, inv, tq);
        } else {
          const int64_t off = (int64_t)(hl * p.G + hq) * p.slots + 2 * cta + (r.first == 0 ? 1 : 0);
          c.store_part(p.ws_o + off * D, r2, inv, tq);
          if (tq == 0) p.ws_lse[off] = c.m_run[r2] + log2f(c.l_run[r2]);
        }
      }
    }
  }
}

// Merge of the rows that several CTAs met in, in token order.  Bound by latency: the statistics of up to 32 parts are read side by
// side, and eight partial rows are requested before the first is added.
template <typename T, int D>
__global__ void flash_decode_shares_merge_kernel(const ShareParams p) {
  pdl_prologue();
  const int b = blockIdx.x, head = blockIdx.y, heads = p.HB * p.G, blk = head / heads, local = head - blk * heads;
  const int2 who = __ldcg(p.ws_info + blk * p.batch + b);   // of shares (else, and of an empty row: an earlier call's)
  const bool splits = __ldcg(p.ws_cut) != 0;
  const int64_t len = load_index(p.seq_len, b, p.len_w);
  T* out = reinterpret_cast<T*>(p.out) + (int64_t)b * p.o_bs + (int64_t)head * p.o_hs + threadIdx.x;
  if (len <= 0) {
    *out = from_f32<T>(0.f);
    return;
  }
  int n = who.y - who.x + 1;
  if (splits) {
    const int64_t all = (len + p.chunk - 1) / p.chunk;
    n = all < p.splits ? (int)all : p.splits;
  } else if (n < 2) {
    return;                                                 // written by its only CTA
  }
  const int64_t base = splits ? ((int64_t)b * p.Hq + head) * p.splits : (int64_t)local * p.slots + 2 * who.x;
  auto part = [&](int i) { return base + (splits ? i : i == 0 ? 1 : 2 * i); };
  if (n == 1) {                                             // most rows of a step far below its bound
    *out = from_f32<T>(__ldcg(p.ws_o + base * D + threadIdx.x));
    return;
  }
  const int lane = threadIdx.x & 31;
  const int d = threadIdx.x;                                // blockDim.x == D
  auto ask = [&](float (&v)[8], int from) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = from + i < n ? __ldcg(p.ws_o + part(from + i) * D + d) : 0.f;
  };
  // the first rows are asked for along with the statistics
  float first[8];
  const float lse0 = lane < n ? __ldcg(p.ws_lse + part(lane)) : -INFINITY;
  ask(first, 0);
  float M = lse0;
  for (int i = lane + 32; i < n; i += 32) M = fmaxf(M, __ldcg(p.ws_lse + part(i)));
  M = warp_reduce_max(M);
  float acc = 0.f, L = 0.f;
  float mine = fast_exp2(lse0 - M);                         // lanes beyond n: 0
  auto add = [&](const float (&v)[8], int from) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float w = __shfl_sync(0xffffffffu, mine, (from + i) & 31);
      if (from + i < n) { acc += w * v[i]; L += w; }
    }
  };
  add(first, 0);
  for (int from = 8; from < n; from += 8) {
    if (from % 32 == 0) mine = from + lane < n ? fast_exp2(__ldcg(p.ws_lse + part(from + lane)) - M) : 0.f;
    float v[8];
    ask(v, from);
    add(v, from);
  }
  *out = from_f32<T>(acc / L);
}

struct Plan { int splits, chunk, qblocks, HB, stages, smem; bool cluster; int share_grid, share_smem; };   // share_grid 0: not the shares' kernel

// ring of a block of HB kv heads: stages and bytes
void plan_ring(Plan& pl, int D, int smem_cap) {
  const int stage = kTT * row_pitch(pl.HB, D);
  int stages = kMaxStages;
  while (stages > 2 && stages * stage > smem_cap) --stages;
  // prefer two resident CTAs per SM when a 3-deep ring fits in half the shared memory
  if (stages * stage > smem_cap / 2 && 3 * stage <= smem_cap / 2) stages = 3;
  pl.stages = stages;
  pl.smem = stages * stage + 128;
}

// Steps of up to 256 tokens a row that leave most of the chip idle: one wave of clusters of eight splits, two of their CTAs to an
// SM.  A tile costs its CTA 0.6 - 1 us (copies, and one warp's chain of products), the merge kernel 3 us, a cluster's launch and
// barriers 2 us.  us in a graph, splits of 64 tokens and the merge kernel -> this: 8 kv heads of 128, one sequence of 200 tokens
// 8.6 -> 6.6, of 80 7.5 -> 5.1, eight of 200 8.8 -> 7.7; 16 of 4 kv heads 8.6 -> 7.4; mixed lengths under that bound 8.6 -> 6.6, 9.2 ->
// 7.3 and 9.4 -> 6.8; rows of a quarter of the bound 8.4 -> 6.2, 8.7 -> 7.1 and 8.9 -> 6.5; of one tile, under 65, 5.1 - 5.9 -> 4.9 - 5.5.
// None of 540 mixtures (1 - 16 sequences, bounds of 65 - 256, six head layouts) is slower.
// Longer splits are the longer chain here (512 tokens in four tiles each 9.1 against 8.9), up to four tiles there is a single
// split without a merge, and with one CTA to an SM the clusters of eight do not all fit (16 sequences of 8 kv heads 8.7 against
// 13.1).
bool plan_cluster(Plan& pl, int64_t batch, int G, int Hkv, int D, int64_t tiles, int hb_cap, int smem_cap) {
  if (tiles <= 4 || tiles > 2 * kMaxCluster) return false;
  Plan c = pl;
  c.HB = 0;
  for (int h = hb_cap; h >= 1; --h)
    if (Hkv % h == 0 && batch * (Hkv / h) * kMaxCluster <= b2l_num_sms()) c.HB = h;
  if (c.HB == 0) return false;
  plan_ring(c, D, smem_cap);
  if (2 * c.smem > smem_cap) return false;
  if ((int64_t)c.HB * G * (D + 1) * 4 > c.smem - 128) return false;     // the partial rows lie over the ring
  c.splits = kMaxCluster;
  c.chunk = (int)((tiles + kMaxCluster - 1) / kMaxCluster) * kTT;
  c.cluster = true;
  pl = c;
  return true;
}

// Steps that would take several waves of CTAs of which an SM holds one or two, whose rings of large stages start anew with each.
// us in a graph, split and merge kernel -> shares: 8 kv heads of 128, 32 sequences of 1000 tokens 36.1 -> 30.3, of 500 - 1000 27.2 ->
// 24.7, of 1000 - 2000 50.7 -> 41.5, 256 of 200 59.1 -> 50.5; 4 kv heads, 32 of 1000 - 2000 29.9 -> 25.8, 64 of 1000 35.4 -> 31.6; 32 kv
// heads of one query head each, whose warps have the most to do per byte, 64 of 250 - 500 94.9 -> 84.8, of 1000 205 -> 204.  The lengths
// are not known here.  Far below the bound the splits that have tokens go to a CTA each, which is level or faster in most (8 kv heads, one
// of 1000 among 31 of 50 11.1 -> 10.5, 32 of 200 11.3 -> 11.1; 4 kv heads, 32 of 40 under 2000 8.7 -> 9.1; 32 kv heads, one of 1600 under
// 8000 13.1 -> 12.5; slowest: 8 kv heads, 8 of 800 under 4000 11.1 -> 12.0, 4 kv heads, one of 2000 among 31 of 100 12.3 -> 13.4).
// Below 13 tiles per CTA, or with more CTAs to an SM, the splits stay: 8 kv heads 32 x 480 16.7 against 16.2, but 64 x 256 16.7 / 17.8,
// 128 x 128 18.1 / 20.6; 2 kv heads of 64, 32 x 2000 13.2 / 20.
void plan_shares(Plan& pl, int64_t batch, int Hkv, int D, int64_t tiles, int smem_cap) {
  if (pl.splits < 2 || D > 128 || batch * tiles * (Hkv / pl.HB) >= (1ll << 26)) return;
  pl.share_smem = pl.smem + (int)(3 * batch + 1) * 4;
  if (pl.share_smem > smem_cap) return;
  int per_sm = (smem_cap + 256) / (pl.share_smem + 1024);
  if (per_sm > 2) return;
  if (per_sm < 1) per_sm = 1;
  if (batch * tiles * (Hkv / pl.HB) < (Hkv > pl.HB ? 6ll : 13ll) * per_sm * b2l_num_sms()) return;
  // One wave: by registers, too, an SM may hold one CTA only, of heads of 128 with two
  // warps of query heads to a kv head (4 kv heads, 20 query heads each, 32 of 1000 - 2000 tokens, splits 53.5 us, shares in two waves
  // 46.4, in one 41.4).
  if (per_sm == 2 && 2 * (pl.HB * pl.qblocks + 1) * 32 * share_regs(D) > 65536) per_sm = 1;
  pl.share_grid = per_sm * b2l_num_sms();
}

// Pure function of host-known sizes => identical inside and outside graph capture.
Plan make_plan(int64_t batch, int Hq, int Hkv, int D, int64_t max_len) {
  Plan pl;
  const int G = Hq / Hkv;
  pl.qblocks = (G + 15) / 16;
  int hb_cap = kMaxConsumers / pl.qblocks;
  if (hb_cap < 1) hb_cap = 1;
  // a 3-stage ring must fit the opt-in shared memory
  const int smem_cap = b2l_max_smem_optin() - 256;
  while (hb_cap > 1 && 3 * kTT * row_pitch(hb_cap, D) > smem_cap) --hb_cap;
  int HB = 1;
  for (int h = 1; h <= hb_cap; ++h)
    if (Hkv % h == 0) HB = h;
  pl.HB = HB;
  plan_ring(pl, D, smem_cap);
  const int64_t pairs = batch * (Hkv / HB);
  const int64_t tiles = max_len > 0 ? (max_len + kTT - 1) / kTT : 1;
  pl.cluster = false;
  pl.share_grid = 0;
  if (plan_cluster(pl, batch, G, Hkv, D, tiles, hb_cap, smem_cap)) return pl;
  // Six CTAs per SM over all splits of the longest possible length.  max_len is only a bound: the lengths are device data, one
  // long sequence may stand among short ones, and a captured graph's bucket may be twice the longest.  One wave of larger
  // splits is faster where every length is near max_len (32 sequences of 1000 - 2000 tokens, 8 kv heads of 128: 25 splits
  // 54 us, 9 splits 47 us) and slower where it is not: sequences shorter than a split then occupy one CTA each.
  const int64_t target = 6LL * b2l_num_sms();
  int64_t splits = (target + pairs - 1) / pairs;
  const int64_t max_splits = (tiles + 3) / 4;   // at least 4 tiles (64 tokens) per split
  if (splits > max_splits) splits = max_splits;
  if (splits < 1) splits = 1;
  const int64_t tiles_per = (tiles + splits - 1) / splits;
  pl.splits = (int)((tiles + tiles_per - 1) / tiles_per);
  pl.chunk = (int)(tiles_per * kTT);
  plan_shares(pl, batch, Hkv, D, tiles, smem_cap);
  return pl;
}
int64_t split_rows(const Plan& pl, int64_t batch, int Hq) { return batch * Hq * pl.splits; }
// partial rows of either cut, and behind them the notes
int64_t share_rows(const Plan& pl, int64_t batch, int Hq, int Hkv) {
  const int64_t shares = 2ll * pl.share_grid * (Hq / Hkv) * pl.HB, splits = split_rows(pl, batch, Hq);
  return shares > splits ? shares : splits;
}
int64_t share_bytes(const Plan& pl, int64_t batch, int Hq, int Hkv, int D) {
  return share_rows(pl, batch, Hq, Hkv) * (D + 1) * 4 + 8 + batch * (Hkv / pl.HB) * 8 + 16;
}

template <typename T, int D>
int launch_decode(const ShareParams& p, const Plan& pl, int64_t batch, cudaStream_t st) {
  if (pl.cluster) {
    static int configured_cluster[64] = {0};
    auto kern = flash_decode_split_kernel<T, D, FD_CLUSTER>;
    B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, pl.smem, configured_cluster));
    b2l_hang_arm(st);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)p.splits, (unsigned)(p.Hkv / p.HB), (unsigned)batch);
    cfg.blockDim = dim3((p.HB * p.qblocks + 1) * 32);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = b2l_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kern, p);
    B2L_LAUNCH_CHECK();
    return B2L_OK;
  }
  if constexpr (D <= 128) {
    if (p.ws_info != nullptr) {
      static int configured_shares[64] = {0};
      auto kern = flash_decode_shares_kernel<T, D>;
      B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, pl.share_smem, configured_shares));
      b2l_launch(kern, dim3((unsigned)pl.share_grid), dim3((p.HB * p.qblocks + 1) * 32), (size_t)pl.share_smem, st, p);
      B2L_LAUNCH_CHECK();
      b2l_launch(flash_decode_shares_merge_kernel<T, D>, dim3((unsigned)batch, (unsigned)p.Hq), dim3(D), (size_t)0, st, p);
      B2L_LAUNCH_CHECK();
      return B2L_OK;
    }
  }
  const bool merge = p.splits > 1 && p.tickets == nullptr;
  static int configured[2][64] = {{0}};
  constexpr int kSplits = D < 256 ? FD_SPLITS : FD_WHOLE;
  auto kern = merge ? flash_decode_split_kernel<T, D, kSplits> : flash_decode_split_kernel<T, D, FD_WHOLE>;
  B2L_CUDA_CHECK(b2l_ensure_dynamic_smem(kern, pl.smem, configured[merge && D < 256]));     // one record per kernel
  dim3 grid((unsigned)p.splits, (unsigned)(p.Hkv / p.HB), (unsigned)batch);
  const int threads = (p.HB * p.qblocks + 1) * 32;
  b2l_launch(kern, dim3(grid), dim3(threads), (size_t)(pl.smem), st, p);
  B2L_LAUNCH_CHECK();
  if (merge) {
    dim3 g2((unsigned)batch, (unsigned)p.Hq);
    // up to nine blocks per SM the merge waits for its rows, beyond that the shorter kernel is the faster one (kv heads of 128,
    // up to 2000 tokens: 24 x 32 heads 44.0 against 40.7 us, 48 x 28 heads 31.7 / 30.6; 64 x 32 heads, 1000 of 4096 59.4 / 60.9)
    if (p.splits > 8 && batch * p.Hq <= 9LL * b2l_num_sms()) b2l_launch(flash_decode_combine_kernel<T, D, true>, dim3(g2), dim3(D >= 128 ? 128 : 64), (size_t)(0), st, p);
    else b2l_launch(flash_decode_combine_kernel<T, D, false>, dim3(g2), dim3(D >= 128 ? 128 : 64), (size_t)(0), st, p);
    B2L_LAUNCH_CHECK();
  }
  return B2L_OK;
}

}  // namespace

// What a call does with these sizes, for tests and tools (no GPU work): out[0..4] = {form: 0 a grid of splits, 1 clusters, 2 shares;
// splits per row; tokens per split; CTAs of the shares' grid; blocks of kv heads}
extern "C" int b2l_flash_decoding_plan(int64_t batch, int num_q_heads, int num_kv_heads, int head_dim, int64_t max_seq_len, int* out,
                                       void* /*reserved*/) {
  B2L_REQUIRE(out && batch > 0 && num_q_heads > 0 && num_kv_heads > 0 && num_q_heads % num_kv_heads == 0, "flash_decoding_plan: bad arguments");
  const Plan pl = make_plan(batch, num_q_heads, num_kv_heads, head_dim, max_seq_len);
  out[0] = pl.cluster ? 1 : pl.share_grid != 0 ? 2 : 0;
  out[1] = pl.splits;
  out[2] = pl.chunk;
  out[3] = pl.share_grid;
  out[4] = num_kv_heads / pl.HB;
  return B2L_OK;
}

extern "C" int64_t b2l_flash_decoding_workspace_bytes(int64_t batch, int num_q_heads, int num_kv_heads, int head_dim,
                                                       int64_t max_seq_len) {
  if (batch <= 0 || num_q_heads <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads != 0) return 0;
  Plan pl = make_plan(batch, num_q_heads, num_kv_heads, head_dim, max_seq_len);
  if (pl.splits <= 1 || pl.cluster) return 16;
  if (pl.share_grid != 0) return share_bytes(pl, batch, num_q_heads, num_kv_heads, head_dim);
  return split_rows(pl, batch, num_q_heads) * (head_dim + 1) * 4 + 16;
}

extern "C" int b2l_flash_decoding(void* out, const void* q, const void* k_cache, const void* v_cache,
                                  const void* b_req_tokens_table, const void* b_req_idx, int req_idx_width,
                                  const void* b_seq_len, int seq_len_width, int64_t batch, int num_q_heads,
                                  int num_kv_heads, int head_dim, int64_t max_seq_len, float qk_scale,
                                  int64_t q_batch_stride, int64_t q_head_stride, int64_t k_token_stride,
                                  int64_t k_head_stride, int64_t v_token_stride, int64_t v_head_stride,
                                  int64_t table_batch_stride, int64_t table_seq_stride, int64_t o_batch_stride,
                                  int64_t o_head_stride, void* workspace, int64_t workspace_bytes, void* tickets,
                                  int64_t num_tickets, int dtype, void* stream) {
  B2L_REQUIRE(out && q && k_cache && v_cache && b_req_tokens_table && b_req_idx && b_seq_len,
              "flash_decoding: null pointer");
  B2L_REQUIRE(num_q_heads > 0 && num_kv_heads > 0 && num_q_heads % num_kv_heads == 0,
              "flash_decoding: num_q_heads (%d) must be a multiple of num_kv_heads (%d)", num_q_heads, num_kv_heads);
  B2L_REQUIRE((req_idx_width == 4 || req_idx_width == 8) && (seq_len_width == 4 || seq_len_width == 8),
              "flash_decoding: index widths must be 4 or 8");
  B2L_REQUIRE(k_token_stride % 8 == 0 && v_token_stride % 8 == 0 && k_head_stride % 8 == 0 && v_head_stride % 8 == 0 &&
                  (uintptr_t)k_cache % 16 == 0 && (uintptr_t)v_cache % 16 == 0,
              "flash_decoding: K/V rows must be 16-byte aligned");
  B2L_REQUIRE(q_head_stride % 2 == 0 && q_batch_stride % 2 == 0 && (uintptr_t)q % 4 == 0 && o_head_stride % 2 == 0 &&
                  o_batch_stride % 2 == 0 && (uintptr_t)out % 4 == 0,
              "flash_decoding: q/out rows must be 4-byte aligned");
  B2L_REQUIRE(head_dim == 32 || head_dim == 64 || head_dim == 128 || head_dim == 256,
              "flash_decoding: head_dim %d (supported: 32, 64, 128, 256)", head_dim);
  if (batch == 0) return B2L_OK;
  Plan pl = make_plan(batch, num_q_heads, num_kv_heads, head_dim, max_seq_len);
  ShareParams p;
  p.q = q; p.q_bs = q_batch_stride; p.q_hs = q_head_stride;
  p.k = k_cache; p.k_ts = k_token_stride; p.k_hs = k_head_stride;
  p.v = v_cache; p.v_ts = v_token_stride; p.v_hs = v_head_stride;
  p.table = (const int32_t*)b_req_tokens_table; p.tab_bs = table_batch_stride; p.tab_ss = table_seq_stride;
  p.req_idx = b_req_idx; p.req_w = req_idx_width;
  p.seq_len = b_seq_len; p.len_w = seq_len_width;
  p.out = out; p.o_bs = o_batch_stride; p.o_hs = o_head_stride;
  p.Hq = num_q_heads; p.Hkv = num_kv_heads; p.G = num_q_heads / num_kv_heads; p.qblocks = pl.qblocks;
  p.HB = pl.HB; p.stages = pl.stages; p.chunk = pl.chunk; p.splits = pl.splits;
  p.scale_log2 = qk_scale * 1.4426950408889634f;
  // how contiguous is one token's K|V for this CTA's head block?
  const bool heads_packed = k_head_stride == head_dim && v_head_stride == head_dim;
  const bool fused_run = heads_packed && pl.HB == num_kv_heads && k_token_stride == v_token_stride &&
                         (const char*)v_cache == (const char*)k_cache + (int64_t)num_kv_heads * head_dim * 2;
  p.copy_mode = fused_run ? 0 : (heads_packed ? 1 : 2);
  p.ws_o = nullptr; p.ws_lse = nullptr; p.ws_info = nullptr;
  p.batch = (int)batch;
  // the split CTAs merge their own results when the caller provides zeroed tickets (one per batch row x head block)
  p.tickets = (tickets && num_tickets >= batch * (num_kv_heads / pl.HB)) ? (int*)tickets : nullptr;
  if (pl.splits > 1 && !pl.cluster) {
    // (room for the splits alone is enough, with its own formula or an earlier one's: the shares then stay out)
    const int64_t rows = split_rows(pl, batch, num_q_heads), need = rows * (head_dim + 1) * 4 + 16;
    B2L_REQUIRE(workspace && workspace_bytes >= need, "flash_decoding: workspace too small (%lld < %lld)",
                (long long)workspace_bytes, (long long)need);
    B2L_REQUIRE((uintptr_t)workspace % 16 == 0, "flash_decoding: workspace must be 16-byte aligned");
    p.ws_o = (float*)workspace;
    p.ws_lse = p.ws_o + rows * head_dim;
    if (pl.share_grid != 0 && p.tickets == nullptr && workspace_bytes >= share_bytes(pl, batch, num_q_heads, num_kv_heads, head_dim)) {
      const int64_t most = share_rows(pl, batch, num_q_heads, num_kv_heads);
      p.slots = 2 * pl.share_grid;
      p.ws_lse = p.ws_o + most * head_dim;
      p.ws_info = (int2*)(p.ws_lse + (most + 1) / 2 * 2);
      p.ws_cut = (int*)(p.ws_info + batch * (num_kv_heads / pl.HB));
    }
  }
  cudaStream_t st = (cudaStream_t)stream;
#define DISPATCH_D(TT)                                                    \
  switch (head_dim) {                                                     \
    case 32: return launch_decode<TT, 32>(p, pl, batch, st);              \
    case 64: return launch_decode<TT, 64>(p, pl, batch, st);              \
    case 128: return launch_decode<TT, 128>(p, pl, batch, st);            \
    default: return launch_decode<TT, 256>(p, pl, batch, st);             \
  }
  if (dtype == B2L_F16) { DISPATCH_D(__half) }
  if (dtype == B2L_BF16) { DISPATCH_D(__nv_bfloat16) }
#undef DISPATCH_D
  B2L_UNSUPPORTED("flash_decoding: dtype %d", dtype);
}
