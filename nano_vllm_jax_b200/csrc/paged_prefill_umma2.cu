// Ragged packed prefill attention on CTA pairs: the tcgen05 tile kernel with `cta_group::2`.
//
// The single-CTA kernel (paged_prefill_umma.cu) is bound by what one SM can take in from L2:
// every 64-key tile costs it 64 KiB for 128 query rows.  Here two CTAs of a cluster (the two
// SMs of a TPC) work on two neighbouring 32-token tiles of the same table row and KV head =
// 256 query rows, and every K/V tile is loaded once for the pair: CTA r keeps keys
// [32 r, 32 r + 32) of the K tile and head dims [128 r, 128 r + 128) of the V tile, 32 KiB per
// tile and SM instead of 64.  `tcgen05.mma.cta_group::2` (issued by CTA 0 alone) multiplies the
// 128 rows each CTA holds in its own tensor memory (Q, later P) with the B operand assembled
// from both halves, and leaves each CTA's 128 x N result in that CTA's tensor memory.
//   S:   M 256 (2 x 128), N 64 keys (2 x 32),  K 16 dims  x 16 per tile
//   P V: M 256,           N 256 dims (2 x 128), K 16 keys x 4 per tile, P as hi + lo
// Roles per CTA as in the single-CTA kernel (warp 0 TMA producer, warp 1 MMA issue in CTA 0,
// warps 2-9 softmax); what crosses the pair:
//   * both producers' TMA loads complete on CTA 0's full barriers (cp.async.bulk.tensor with
//     .cta_group::2 and the barrier address of rank 0); no load is a multicast;
//   * `tcgen05.commit` with a two-CTA mask releases K/V stages and hands scores over in both CTAs;
//   * the softmax warps of both CTAs arrive on CTA 0's "Q staged", "S read" and "P written" barriers.
// A cluster barrier after set-up and one before the tensor memory is freed fence the pair.
// Every mbarrier wait is bounded; a timeout flags NVJ_DEV_TIMEOUT and both CTAs still reach
// the final cluster barrier and free their tensor memory.
// Short batches (a 512-token chunk is 18 CTA pairs on 74 pair slots) split every tile's key range over up to kU2MaxSplits pairs
// (blockIdx.z), which form one cluster: each leaves its un-normalised rows and their (max, sum) in its shared memory, and
// behind a cluster barrier every CTA folds its share of the rows out of all of them and writes it.  (The splits used to go through
// a workspace and a second launch that folded them: 128 KiB written and read again per CTA, and 4 us; the chunk behind 1024
// cached tokens 23.8 -> 21.9 us, 64 tokens behind 400 18.5 -> 16.3.)
// Semantics: nanovllm_jax/kv_cache.py:831-849, nanovllm_jax/kernels/full_attention_triton.py:51-145.

#include <cstddef>

#include "cluster.cuh"
#include "paged_decode.cuh"
#include "umma.cuh"

namespace nvj {

constexpr int kU2Tokens = 32;    // query tokens per CTA (64 per pair)
constexpr int kU2Rows = 128;     // query rows per CTA
constexpr int kU2Keys = 64;      // keys per tile
constexpr int kU2Stages = 4;
constexpr int kU2Threads = 320;
constexpr int kU2SoftmaxThreads = 256;
constexpr int kU2TmemCols = 512;
constexpr int kU2ColQ = 0, kU2ColS = 128, kU2ColP = 192, kU2ColO = 256;  // queries, scores, weights (hi, lo), output
constexpr uint32_t kU2TileBytes = kU2Keys * kRowBytes;  // a whole K (or V) tile: both CTAs' halves, 32 KiB
constexpr uint32_t kU2LeaderMask = 0xFEFFFFFFu;         // clears the CTA-rank bit of a shared::cluster address
constexpr float kU2Log2e = 1.4426950408889634f;
constexpr float kU2RescaleGap = 8.f;
constexpr int kU2MaxSplits = 4;
// A key tile costs a pair ~1 us, a split the barrier and the fold, ~2 us.  Key ranges of kU2SplitFrom tiles or more are split into
// pieces of at least kU2MinSplitTiles tiles: from 4 on 100 tokens behind 220 take 18.7 us instead of 16.9, from 8 on 64 behind 400
// 19.0 instead of 16.3 and 400 behind none 18.4 instead of 17.4.  Four pieces only while the pairs' clusters of eight CTAs all fit
// (15 here): a tile of 16 - 18 pairs and heads gets three (512 tokens behind 3584: 39.5 us, 36.6 with four and a second launch).
constexpr int kU2SplitFrom = 6;
constexpr int kU2MinSplitTiles = 2;

// Development aid, compiled in only with -DNVJ_PHASE_TIMING: the first softmax thread of every CTA stamps the global
// timer at the kernel's phase boundaries (slot 7: the number of key tiles), nvj_debug_prefill_phase_ns copies them out.
#ifdef NVJ_PHASE_TIMING
__device__ unsigned long long g_u2_phase_ns[512][8];
#define NVJ_U2_PHASE(i) do { if (threadIdx.x == 64) g_u2_phase_ns[(blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x & 511][i] = global_timer_ns(); } while (0)
#define NVJ_U2_NOTE(i, v) do { if (threadIdx.x == 64) g_u2_phase_ns[(blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x & 511][i] = (v); } while (0)
#else
#define NVJ_U2_PHASE(i) do { } while (0)
#define NVJ_U2_NOTE(i, v) do { } while (0)
#endif

struct Umma2Params {
  const void* q;
  const int32_t* block_tables;
  const int32_t* kv_lens;
  const int32_t* positions;
  const int32_t* query_start_loc;
  float* out;
  int32_t* status;
  long long num_blocks;
  int rows, token_bucket, table_width, skip_single, q_dtype;
  int counted;    // 1: the launch has exactly the caller's number of pairs plus an idle one; more pairs are flagged
  int32_t* beside;  // nullable: set once what lies in front of this grid is visible (DecodeParams::beside)
  int zero_fill;  // 1: the kernel itself zeroes what no tile writes (padding tokens, rows of several tokens without keys)
  int split_p;  // 1: P enters P V as two bf16 terms (hi + lo), 0: as one (the weights are then bf16-rounded)
  float scale;
  // key-range splits (gridDim.z > 1)
  int pair_slots;  // CTA pairs that run at once
};

struct Umma2Smem {
  alignas(1024) char k[kU2Stages][2][8192];  // [stage][this CTA's two blocks][8-key group][64-d chunk][8 keys][128 B]
  alignas(1024) char v[kU2Stages][4][4096];  // [stage][block][8-key group][this CTA's two 64-d chunks][8 keys][128 B]
  // used in CTA 0 only: q_full, k_full, v_full, s_read, p_full; used in both: the rest
  alignas(8) unsigned long long q_full, k_full[kU2Stages], v_full[kU2Stages], k_empty[kU2Stages], v_empty[kU2Stages],
      s_full[2], s_read, o_full;  // s_full: [tile & 1]; o_full: every product has retired
  unsigned long long p_full[2], pv_done[2][2];  // per half of a tile's keys: weights written; the product that reads them retired [tile & 1]
  unsigned long long m_full[4][2];  // per quarter of the rows: the reference of an even / odd tile has been settled
  float m_row[2][kU2Rows];          // the reference itself [tile & 1]
  float2 sums[2][kU2Rows];          // at the end: each group's (reference, sum of weights)
  // this CTA's query rows on their way into tensor memory: [token][head of the group][32 pieces of 16 B], the pieces
  // of token t stored at (piece ^ (t & 7)) so that both the row-wise fill and the token-wise read are conflict-free
  alignas(16) char qstage[kU2Tokens * kG * kD * 2];
  float2 own_ml[kU2Rows];  // this split's (max, sum) per row, for the fold
  uint32_t tmem_base;
  int abort_flag;
};

// ---- cta_group::2 wrappers ---------------------------------------------------------------------
__device__ __forceinline__ void tmem2_alloc(uint32_t smem_dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem2_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[256 x N] (+)= A[256 x 16] B[16 x N] over the CTA pair: each CTA's 128 rows of A and D in its own tensor
// memory at the same addresses, each CTA's N / 2 columns of B in its own shared memory at the same offsets
__device__ __forceinline__ void umma2_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
// arrives, once the MMAs issued so far have retired, on the barrier at this offset in both CTAs of the pair (ranks 2 z and 2 z + 1
// of the cluster)
__device__ __forceinline__ void umma2_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((uint16_t)(3u << (2 * blockIdx.z))) : "memory");
}
// One box of a grouped view into this CTA's shared memory; the bytes are counted on CTA 0's barrier at `bar`'s offset.
__device__ __forceinline__ void tma2_load_5d(uint32_t dst, const CUtensorMap* map, int chunk, int group, int kvh, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3, %4, %5}], [%6];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(chunk), "r"(group), "r"(kvh), "r"(bar & kU2LeaderMask)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
  // default semantics (release at CTA scope): what the arrival publishes lives in tensor memory and is ordered by
  // tcgen05.wait::st + tcgen05.fence; a cluster-scope release here cost ~1700 cycles per arrival
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar & kU2LeaderMask) : "memory");
}
// One arrival for a warp, once all of its lanes have come here.
__device__ __forceinline__ void u2_arrive_warp(uint32_t bar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive_leader(bar);
}
// Instruction descriptor, kind::f16, fp32 accumulate, bf16 A and B, M = 256 over the pair.
__device__ __forceinline__ constexpr uint32_t umma2_idesc(int n, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((256u >> 4) << 24);
}

// ---- warp 0 of both CTAs: TMA loads of this CTA's halves ------------------------------------
__device__ __forceinline__ void u2_producer(const CUtensorMap* k_map, const CUtensorMap* v_map, const Umma2Params& p,
                                            Umma2Smem& sm, int row, int kvh, int kv_len, int tile0, int n_tiles, int rank,
                                            int lane, int first_ids) {
  const int need_blocks = (kv_len + kBlk - 1) / kBlk;
  const int oob = (int)(p.num_blocks * (kBlk / 8));  // a box that starts here is filled with zeros
  int ids = -1;
  for (int t = 0; t < n_tiles; ++t) {
    const int s = t % kU2Stages;
    const uint32_t reuse_parity = ((t / kU2Stages) - 1) & 1;
    if ((t & 7) == 0) {  // block ids of the next 8 tiles, one per lane
      const int bi = (tile0 + t) * 4 + lane;
      ids = -1;
      if (bi < need_blocks && bi < p.table_width) {
        ids = t == 0 ? first_ids : p.block_tables[(long long)row * p.table_width + bi];  // the first eight tiles' came early
        if (ids < 0 || ids >= p.num_blocks) {
          if (rank == 0) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
          ids = -1;
        }
      }
    }
    int z[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int id = __shfl_sync(0xffffffffu, ids, (t & 7) * 4 + b);
      z[b] = id >= 0 ? id * (kBlk / 8) : oob;
    }
    if (t >= kU2Stages && !um_wait(&sm.k_empty[s], reuse_parity, &sm.abort_flag, p.status)) break;
    if (lane == 0) {
      const uint32_t kb = smem_u32(&sm.k_full[s]);
      if (rank == 0) mbar_arrive_expect_tx(kb, kU2TileBytes);  // both CTAs' halves are counted here
#pragma unroll
      for (int b2 = 0; b2 < 2; ++b2)  // this CTA's keys: cache blocks 2 rank, 2 rank + 1 of the tile
        tma2_load_5d(smem_u32(&sm.k[s][b2][0]), k_map, 0, rank ? z[2 + b2] : z[b2], kvh, kb);
    }
    if (t >= kU2Stages && !um_wait(&sm.v_empty[s], reuse_parity, &sm.abort_flag, p.status)) break;
    if (lane == 0) {
      const uint32_t vb = smem_u32(&sm.v_full[s]);
      if (rank == 0) mbar_arrive_expect_tx(vb, kU2TileBytes);
#pragma unroll
      for (int b = 0; b < 4; ++b)  // all keys, this CTA's head dims: 64-d chunks 2 rank, 2 rank + 1
        tma2_load_5d(smem_u32(&sm.v[s][b][0]), v_map, 2 * rank, z[b], kvh, vb);
    }
    __syncwarp();
  }
}

// ---- warp 1 of CTA 0: MMA issue for the pair -------------------------------------------------
// S(t + 2) is issued as soon as the softmax has read S(t + 1), in front of P V(t), which waits for its weights half a tile at a time.  From
// its scores to its weights a tile takes ~2000 cycles, its products 1640: with one tile of scores ahead (and all softmax
// warps on the same tile) a lone pair took 1.02 us per tile, now 0.93; one tile ahead with two softmax groups, or with the weights in
// halves as well, still 1.02.  1000 tokens behind 4000 56.8 -> 51.6 us, 2000 of four prompts 25.5 -> 23.8, 512 behind 1024 21.1 -> 20.0; under the
// power cap, 16384 of one prompt, 1145 -> 1138.
__device__ __forceinline__ bool u2_issue_s(Umma2Smem& sm, const Umma2Params& p, uint32_t tmem, uint64_t k_desc0, int t,
                                           int stage, uint32_t full_parity) {
  if (!um_wait(&sm.k_full[stage], full_parity, &sm.abort_flag, p.status)) return false;
  if (t > 0 && !um_wait(&sm.s_read, (t - 1) & 1, &sm.abort_flag, p.status)) return false;
  tc_fence_after_sync();
  if (um_elect_one()) {
    constexpr uint32_t idesc = umma2_idesc(kU2Keys, false);
    const uint64_t k_desc = k_desc0 + (uint64_t)((stage * (int)sizeof(sm.k[0])) >> 4);
#pragma unroll
    for (int ks = 0; ks < 16; ++ks)  // 16 dims per MMA: 8 columns of Q; K chunk ks / 4, 32 bytes into its swizzled rows
      umma2_bf16_ts(tmem + kU2ColS, tmem + kU2ColQ + ks * 8, k_desc + (uint64_t)(((ks >> 2) * (8 * 128) + (ks & 3) * 32) >> 4), idesc,
                    ks > 0 ? 1u : 0u);
    umma2_commit_pair(smem_u32(&sm.s_full[t & 1]));
    umma2_commit_pair(smem_u32(&sm.k_empty[stage]));
  }
  __syncwarp();
  return true;
}

__device__ __forceinline__ void u2_mma_warp(Umma2Smem& sm, const Umma2Params& p, uint32_t tmem, int n_tiles) {
  const uint64_t k_desc0 = umma_desc(smem_u32(&sm.k[0][0][0]), 16, 4 * 8 * 128);       // keys are rows, groups of 8 4 KiB apart
  const uint64_t v_desc0 = umma_desc(smem_u32(&sm.v[0][0][0]), 8 * 128, 2 * 8 * 128);  // 64-d chunks 1 KiB apart, groups of 8 keys 2
  if (!um_wait(&sm.q_full, 0, &sm.abort_flag, p.status)) return;
  auto scores = [&](int t) { return t >= n_tiles || u2_issue_s(sm, p, tmem, k_desc0, t, t % kU2Stages, (t / kU2Stages) & 1); };
  if (!scores(0) || !scores(1)) return;
  for (int t = 0; t < n_tiles; ++t) {
    if (!scores(t + 2)) return;
    const int sv = t % kU2Stages;
    if (!um_wait(&sm.v_full[sv], (t / kU2Stages) & 1, &sm.abort_flag, p.status)) return;
    constexpr uint32_t idesc = umma2_idesc(kD, true);
    const uint64_t v_desc = v_desc0 + (uint64_t)((sv * (int)sizeof(sm.v[0])) >> 4);
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // 32 keys: their columns are free again while the other half is multiplied
      if (!um_wait(&sm.p_full[h], t & 1, &sm.abort_flag, p.status)) return;
      tc_fence_after_sync();
      if (um_elect_one()) {
#pragma unroll
        for (int kk = 2 * h; kk < 2 * h + 2; ++kk) {  // 16 keys per MMA: 8 columns of P, two 8-key groups of V
          const uint64_t dv = v_desc + (uint64_t)((kk * 4096) >> 4);
          umma2_bf16_ts(tmem + kU2ColO, tmem + kU2ColP + kk * 8, dv, idesc, (t > 0 || kk > 0) ? 1u : 0u);
          if (p.split_p) umma2_bf16_ts(tmem + kU2ColO, tmem + kU2ColP + 32 + kk * 8, dv, idesc, 1u);
        }
        umma2_commit_pair(smem_u32(&sm.pv_done[t & 1][h]));
        if (h == 1) {
          umma2_commit_pair(smem_u32(&sm.v_empty[sv]));
          if (t == n_tiles - 1) umma2_commit_pair(smem_u32(&sm.o_full));
        }
      }
      __syncwarp();
    }
  }
}

// The walk over the key tiles for one softmax thread (row r).  The eight warps are two groups that take the even and the odd tiles,
// a thread a whole row of 64 scores: out of tensor memory, masked, weights back into tensor memory.  What a tile costs from its
// scores to its weights (~2000 cycles: barriers, the trips to tensor memory, 64 exponentials per row) is longer than its products
// (1640), so two tiles have to be on their way.  (With each tile shared by all eight warps, half a row per thread, a lone pair took
// 2050 cycles per tile.)  What stays in turn is the row's reference (the running maximum, moved only when a tile exceeds it
// by 2^kU2RescaleGap): a group settles its tile's reference behind the other's, before its exponentials.  False when a
// wait ran out (the caller still joins its barriers).
__device__ __forceinline__ bool u2_softmax_tiles(Umma2Smem& sm, const Umma2Params& p, uint32_t my_tmem, int tok0, int ntok,
                                                 int kv_len, int tile0, int n_tiles, int group, int r, int token, float& m_row,
                                                 float& l_row) {
  const int my_pos = token < ntok ? p.positions[tok0 + token] : -1;
  const int last_key = my_pos < kv_len - 1 ? my_pos : kv_len - 1;
  const float scale_log2 = p.scale * kU2Log2e;
  const int quarter = r >> 5;
  for (int t = group; t < n_tiles; t += 2) {
    const uint32_t mine = (t >> 1) & 1, before = ((t - 1) >> 1) & 1;  // parities of this tile's and the tile before's barriers
    if (!um_wait(&sm.s_full[group], mine, &sm.abort_flag, p.status)) return false;
    if (t == 0) NVJ_U2_PHASE(3);
    tc_fence_after_sync();
    float s[kU2Keys];
    tmem_ld64(my_tmem + kU2ColS, s);
    tc_fence_before_sync();
    u2_arrive_warp(smem_u32(&sm.s_read));
    const int lim = last_key - (tile0 + t) * kU2Keys;
    float tmax = -INFINITY;
    if (lim >= kU2Keys - 1) {
#pragma unroll
      for (int i = 0; i < kU2Keys; i += 2) tmax = fmaxf(tmax, fmaxf(s[i], s[i + 1]));
    } else {
#pragma unroll
      for (int i = 0; i < kU2Keys; ++i) { s[i] = i <= lim ? s[i] : -INFINITY; tmax = fmaxf(tmax, s[i]); }
    }
    tmax *= scale_log2;  // scale > 0
    float m_new = tmax;
    if (t > 0) {
      if (!um_wait(&sm.m_full[quarter][group ^ 1], before, &sm.abort_flag, p.status)) return false;
      m_new = sm.m_row[group ^ 1][r];
      if (__any_sync(0xffffffffu, tmax > m_new + kU2RescaleGap)) {
        if (!um_wait(&sm.pv_done[group ^ 1][1], before, &sm.abort_flag, p.status)) return false;
        tc_fence_after_sync();
        const float m_old = m_new;
        m_new = fmaxf(m_old, tmax);
        const float f = m_new == -INFINITY ? 1.f : ex2_approx(m_old - m_new);
#pragma unroll 1
        for (int cc = 0; cc < kD / 32; ++cc) {
          float o[32];
          tmem_ld32(my_tmem + kU2ColO + cc * 32, o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] *= f;
          tmem_st32(my_tmem + kU2ColO + cc * 32, o);
        }
      }
    }
    if (t + 1 < n_tiles) {  // the other group's next tile
      sm.m_row[group][r] = m_new;
      __syncwarp();
      if ((r & 31) == 0) mbar_arrive(smem_u32(&sm.m_full[quarter][group]));
    }
    if (m_new != m_row) {  // (this group's first tile included: no weights so far)
      l_row *= m_new == -INFINITY ? 1.f : ex2_approx(m_row - m_new);
      m_row = m_new;
    }
    const float neg_m = m_row == -INFINITY ? 0.f : -m_row;
    uint32_t hi[2][16], lo[2][16];
    const float2 c2 = make_float2(scale_log2, scale_log2), m2 = make_float2(neg_m, neg_m);
#pragma unroll
    for (int e = 0; e < kU2Keys / 2; ++e) {  // two keys at a time, packed fp32 arithmetic
      float2 w = fma2(make_float2(s[2 * e], s[2 * e + 1]), c2, m2);
      w.x = ex2_approx(w.x);
      w.y = ex2_approx(w.y);
      // One running sum per thread: even and odd keys apart, added at the end, measured a 20% larger error on peaked scores.  (The two
      // groups' sums, over the even and the odd tiles, are added at the end without one: 1.257e-6 before as after.)
      l_row += w.x + w.y;
      const __nv_bfloat162 h = __floats2bfloat162_rn(w.x, w.y);
      const float2 rest = fma2(make_float2(__low2float(h), __high2float(h)), make_float2(-1.f, -1.f), w);  // exact
      const __nv_bfloat162 g = __floats2bfloat162_rn(rest.x, rest.y);
      hi[e >> 4][e & 15] = *reinterpret_cast<const uint32_t*>(&h);
      lo[e >> 4][e & 15] = *reinterpret_cast<const uint32_t*>(&g);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // as soon as P V of the tile before has read this half of its weights
      if (t >= 1 && !um_wait(&sm.pv_done[group ^ 1][h], before, &sm.abort_flag, p.status)) return false;
      tmem_st16(my_tmem + kU2ColP + h * 16, hi[h]);
      if (p.split_p) tmem_st16(my_tmem + kU2ColP + 32 + h * 16, lo[h]);
      tmem_st_wait();
      tc_fence_before_sync();
      u2_arrive_warp(smem_u32(&sm.p_full[h]));
    }
  }
  return true;
}

// The tile's query rows, 2 KiB per token (the group's four heads lie side by side), as whole 512-byte rows per warp
// instruction, all sixteen loads of a thread in flight at once: softmax warp sw takes tokens 4 sw .. 4 sw + 3.
__device__ __forceinline__ void u2_request_q(const Umma2Params& p, int tok0, int ntok, int kvh, int warp, int lane, uint4 (&u)[4][4]) {
  const int sw = (warp - 2) & 7;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int tk = sw * 4 + a;
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.q) +
                                                      ((long long)(tok0 + tk) * kHq + kvh * kG) * kD) + lane;
#pragma unroll
    for (int h = 0; h < 4; ++h) u[a][h] = tk < ntok ? ld_stream_u4(src + h * 32) : make_uint4(0u, 0u, 0u, 0u);
  }
}

// Where the 16-byte piece `c` of row `r` of the output tile lies in the freed stages, in floats.
__device__ __forceinline__ int u2_piece(int r, int c) { return r * kD + (((c & ~7) | ((c ^ r) & 7)) << 2); }

// ---- warps 2-9 of both CTAs: Q staging, softmax, epilogue for this CTA's 128 rows -------------
__device__ __forceinline__ void u2_softmax_warps(Umma2Smem& sm, const Umma2Params& p, uint32_t tmem, int tok0, int ntok,
                                                 int kvh, int kv_len, int tile0, int n_tiles, int splits, int warp, int lane,
                                                 const uint4 (&u)[4][4]) {
  const int quarter = warp & 3, half = (warp - 2) >> 2;
  const int r = quarter * 32 + lane, token = lane, hl = quarter;
  const uint32_t my_tmem = tmem + ((uint32_t)(quarter * 32) << 16);
  if (p.q_dtype == NVJ_BF16) {
    // The tile's query rows (`u`, requested by u2_request_q before the pair was set up) go through shared memory: a
    // thread that fetched its own row directly would touch 32 lines per instruction and wait for memory four times
    // in a row (4.4 us of a 30 us kernel on a 512-token chunk).
    const int sw = (warp - 2) & 7;  // 0..7: four tokens each
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int tk = sw * 4 + a;
#pragma unroll
      for (int h = 0; h < 4; ++h)
        *reinterpret_cast<uint4*>(sm.qstage + tk * 2048 + h * 512 + ((lane ^ (tk & 7)) << 4)) = u[a][h];
    }
    named_bar_sync(1, kU2SoftmaxThreads);
    // this row's half of Q (128 dims) -> 64 TMEM columns, two bf16 per column
    const char* mine = sm.qstage + token * 2048 + hl * 512;
#pragma unroll 1
    for (int part = 0; part < 4; ++part) {
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint4 x = *reinterpret_cast<const uint4*>(mine + (((half * 16 + part * 4 + i) ^ (token & 7)) << 4));
        w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
      }
      tmem_st16(my_tmem + kU2ColQ + half * 64 + part * 16, w);
    }
    tmem_st_wait();
    tc_fence_before_sync();
    u2_arrive_warp(smem_u32(&sm.q_full));
    NVJ_U2_PHASE(2);
  } else {  // fp32 queries: every thread converts its own row
    const long long qrow = ((long long)(tok0 + token) * kHq + kvh * kG + hl) * kD + half * (kD / 2);
#pragma unroll 1
    for (int part = 0; part < 4; ++part) {
      uint32_t w[16];
      if (token >= ntok) {
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = 0u;
      } else {
        const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(p.q) + qrow + part * 32);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 f = src[i];
          const __nv_bfloat162 a = __floats2bfloat162_rn(f.x, f.y), b2 = __floats2bfloat162_rn(f.z, f.w);
          w[2 * i] = *reinterpret_cast<const uint32_t*>(&a);
          w[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&b2);
        }
      }
      tmem_st16(my_tmem + kU2ColQ + half * 64 + part * 16, w);
    }
    tmem_st_wait();
    tc_fence_before_sync();
    u2_arrive_warp(smem_u32(&sm.q_full));
    NVJ_U2_PHASE(2);
  }
  float m_row = -INFINITY, l_row = 0.f;
  bool alive = u2_softmax_tiles(sm, p, my_tmem, tok0, ntok, kv_len, tile0, n_tiles, half, r, token, m_row, l_row);
  // ---- epilogue.  From here on the softmax threads meet at CTA-wide named barriers, so a thread whose wait ran out
  // does not leave: it skips the work and everybody returns together once the barrier has made the flag visible.
  NVJ_U2_PHASE(4);
  sm.sums[half][r] = make_float2(m_row, l_row);
  named_bar_sync(2 + quarter, 64);  // the quarter's two warps
  {  // the last tile's group holds the row's reference (they grow); the other's sum comes to it
    const float2 other = sm.sums[half ^ 1][r];
    const float m = fmaxf(m_row, other.x);
    const float mine = m == -INFINITY ? 0.f : ex2_approx(m_row - m) * l_row, others = m == -INFINITY ? 0.f : ex2_approx(other.x - m) * other.y;
    m_row = m;
    l_row = half == 0 ? mine + others : others + mine;  // (the same in both)
  }
  if (alive) alive = um_wait(&sm.o_full, 0, &sm.abort_flag, p.status);
  tc_fence_after_sync();
  const float inv = splits > 1 ? 1.f : (l_row > 0.f ? 1.f / l_row : 0.f);  // a split leaves its rows un-normalised
  if (splits > 1 && half == 0) sm.own_ml[r] = make_float2(m_row, l_row);
  // The K and V stages (128 KiB, contiguous) are free now: every copy has landed and every product has retired.  The
  // normalised rows are laid down there, [row][256 floats] with the 16-byte pieces of row r stored at (piece ^ (r & 7))
  // inside their group of eight, and leave as whole 512-byte runs per warp instruction.  (Stored straight from the
  // registers, a warp instruction touched 32 lines: 5.4 us of a 30 us kernel on a 512-token chunk.)
  float* stage = reinterpret_cast<float*>(&sm.k[0][0][0]);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the stages were last written by bulk copies
  static_assert(sizeof(sm.k) + sizeof(sm.v) >= (size_t)kU2Rows * kD * sizeof(float) && offsetof(Umma2Smem, v) == sizeof(sm.k),
                "the output tile is staged across the K and V stages");
#pragma unroll 1
  for (int cc = 0; cc < kD / 64 && alive; ++cc) {
    float o[32];
    tmem_ld32(my_tmem + kU2ColO + half * (kD / 2) + cc * 32, o);
    const int c0 = (half * (kD / 2) + cc * 32) >> 2;  // first 16-byte piece of these 32 floats within the row
#pragma unroll
    for (int i = 0; i < 8; ++i)
      *reinterpret_cast<float4*>(stage + r * kD + ((c0 + (i ^ (r & 7))) << 2)) =
          make_float4(o[4 * i] * inv, o[4 * i + 1] * inv, o[4 * i + 2] * inv, o[4 * i + 3] * inv);
  }
  named_bar_sync(1, kU2SoftmaxThreads);
  if (*reinterpret_cast<volatile int*>(&sm.abort_flag)) return;  // somebody gave up: the same answer in every thread
  const int sw = (warp - 2) & 7;
  if (splits > 1) return;  // u2_fold_splits takes the rows from here
#pragma unroll 4
  for (int a = 0; a < kU2Rows / 8; ++a) {
    const int rr = sw * (kU2Rows / 8) + a, tk = rr & 31, hd = rr >> 5;
    if (tk >= ntok) continue;
    const long long g = (long long)(tok0 + tk) * kHq + kvh * kG + hd;
#pragma unroll
    for (int h2 = 0; h2 < 2; ++h2) {
      const int c = h2 * 32 + lane;
      reinterpret_cast<float4*>(p.out + g * kD)[c] = *reinterpret_cast<const float4*>(stage + u2_piece(rr, c));
    }
  }
  NVJ_U2_PHASE(5);
}

// The splits' rows, staged by all of them (the same 128 rows in the CTAs of this rank of every pair), into the output: split z of n
// takes rows [128 z / n, 128 (z + 1) / n), a warp the same number of rows one behind the other, two at a time, every split's pieces
// requested before anything is used.  The (max, sum) pairs of a warp's rows come in one load: what counts between the CTAs is the number of
// requests, and with a load of its own for every row the fold took 3.8 us instead of 3.1 (512 tokens behind 1024: 20.2 -> 19.2 us, behind 256
// 17.7 -> 16.5, 64 behind 400 16.1 -> 15.3).  Three rows at a time, or half rows: no faster.
// Returns what cl_sync_read() asks for.
__device__ __forceinline__ bool u2_fold_splits(const Umma2Smem& sm, const Umma2Params& p, int tok0, int ntok, int kvh, int rank, int splits,
                                               int warp, int lane) {
  const float* stage = reinterpret_cast<const float*>(&sm.k[0][0][0]);
  constexpr int kWarps = kU2Threads / 32;
  static_assert((kU2Rows / 2 + kWarps - 1) / kWarps * kU2MaxSplits <= 32, "a warp's rows and their splits are its lanes");
  const int row0 = (int)blockIdx.z * kU2Rows / splits, row1 = ((int)blockIdx.z + 1) * kU2Rows / splits;
  const int per = (row1 - row0 + kWarps - 1) / kWarps, first = row0 + warp * per, last = first + per < row1 ? first + per : row1;
  float w;  // lane 4 i + s: split s's normalised weight in row first + i
  {
    const int s = lane & (kU2MaxSplits - 1), rr = first + lane / kU2MaxSplits;
    float2 e = make_float2(-INFINITY, 0.f);
    if (rr < last && s < splits) e = cl_ld2(cl_map(&sm.own_ml[rr], 2 * s + rank));
    float big = e.x;
#pragma unroll
    for (int o = 1; o < kU2MaxSplits; o <<= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    w = e.x == -INFINITY ? 0.f : ex2_approx(e.x - big);
    float total = w * e.y;
#pragma unroll
    for (int o = 1; o < kU2MaxSplits; o <<= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    w = total > 0.f ? w / total : 0.f;
  }
  bool odd = !(w <= 1.f);
  for (int r0 = first; r0 < last; r0 += 2) {
    float4 x[2][kU2MaxSplits][2];
    bool real[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int rr = r0 + k;
      real[k] = rr < last && (rr & 31) < ntok;
#pragma unroll
      for (int s = 0; s < kU2MaxSplits; ++s)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          x[k][s][h] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (real[k] && s < splits) x[k][s][h] = cl_ld4(cl_map(stage + u2_piece(rr, h * 32 + lane), 2 * s + rank));
        }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (!real[k]) continue;
      const int rr = r0 + k;
      float4* dst = reinterpret_cast<float4*>(p.out + ((long long)(tok0 + (rr & 31)) * kHq + kvh * kG + (rr >> 5)) * kD);
      float4 acc[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll
      for (int s = 0; s < kU2MaxSplits; ++s) {
        const float ws = __shfl_sync(0xffffffffu, w, (rr - first) * kU2MaxSplits + s);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          acc[h].x = fmaf(x[k][s][h].x, ws, acc[h].x); acc[h].y = fmaf(x[k][s][h].y, ws, acc[h].y);
          acc[h].z = fmaf(x[k][s][h].z, ws, acc[h].z); acc[h].w = fmaf(x[k][s][h].w, ws, acc[h].w);
        }
      }
      odd |= cl_not_finite(acc[0]) || cl_not_finite(acc[1]);
      dst[lane] = acc[0];
      dst[32 + lane] = acc[1];
    }
  }
  return odd;
}

// Which (table row, 32-token tile) the CTA with cluster index `cluster` of `clusters` and rank `rank` serves: the
// heaviest pairs (the last tokens of a row see the most keys) get the lowest cluster indices.  Every warp runs this for itself, 32 rows
// at a time (one thread walking the rows paid a trip to the L2 for each: 7 of 24 us on a batch of 32 decode rows and two
// chunks); a row's length and whether any is long enough to be split come with the same trip.  row < 0: no tile (`idle` then numbers
// the clusters beyond the last pair 0, 1, ...).  `total` (the batch's number of pairs) and `any_long` are complete only when `need_total`.
struct U2Tile {
  int row, tok0, ntok, pair_last_tok, kv_len, idle, total;
  bool any_long;
};
__device__ __forceinline__ U2Tile u2_find_tile(const Umma2Params& p, int cluster, int clusters, int rank, bool need_total, int lane) {
  U2Tile t{-1, 0, 0, 0, 0, -1, 0, false};
  int idx = clusters - 1 - cluster;
  for (int base = 0; base < p.rows && (need_total || t.row < 0); base += 32) {
    const int r = base + lane;
    int lo = 0, hi = 0, pairs = 0, len = 0;
    if (r < p.rows) {
      lo = p.query_start_loc[r];
      const int end = p.query_start_loc[r + 1];
      len = p.kv_lens[r];
      hi = end < p.token_bucket ? end : p.token_bucket;
      pairs = hi > lo ? (hi - lo + 2 * kU2Tokens - 1) / (2 * kU2Tokens) : 0;
      if (p.skip_single && end - lo == 1) pairs = 0;
    }
    int incl = pairs;  // pairs of this lane's row and the ones before it in the group
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    const int group = __shfl_sync(0xffffffffu, incl, 31);
    t.total += group;
    if (need_total) t.any_long |= __any_sync(0xffffffffu, len > (kU2SplitFrom - 1) * kU2Keys) != 0;
    if (t.row >= 0) continue;
    const unsigned hit = __ballot_sync(0xffffffffu, idx >= incl - pairs && idx < incl);
    if (hit == 0) {
      idx -= group;
      continue;
    }
    const int at = __ffs(hit) - 1;
    const int row_lo = __shfl_sync(0xffffffffu, lo, at), row_hi = __shfl_sync(0xffffffffu, hi, at);
    const int pair = idx - __shfl_sync(0xffffffffu, incl - pairs, at);
    t.kv_len = __shfl_sync(0xffffffffu, len, at);
    t.row = base + at;
    t.tok0 = row_lo + (2 * pair + rank) * kU2Tokens;
    t.ntok = row_hi - t.tok0 < kU2Tokens ? row_hi - t.tok0 : kU2Tokens;
    if (t.ntok < 0) t.ntok = 0;
    const int pair_end = row_lo + (2 * pair + 2) * kU2Tokens;
    t.pair_last_tok = (pair_end < row_hi ? pair_end : row_hi) - 1;
  }
  if (t.row < 0) t.idle = idx;
  return t;
}
// Key tiles of the pair (warp-collective; the same in every warp of both CTAs): the token of the pair that sees the most
// keys bounds the key range (positions need not grow along the tiles).  `seen`: the larger position of this lane's two tokens.
__device__ __forceinline__ int u2_last_positions(const Umma2Params& p, const U2Tile& t, int rank, int lane) {
  const int tok0 = t.tok0 - rank * kU2Tokens, n = t.pair_last_tok - tok0 + 1;
  const int a = lane < n ? ld_in_turn(p.positions + tok0 + lane) : -1, b = lane + 32 < n ? ld_in_turn(p.positions + tok0 + lane + 32) : -1;
  return a > b ? a : b;
}
__device__ __forceinline__ int u2_key_tiles(int seen, int kv_len) {
  const int max_pos = __reduce_max_sync(0xffffffffu, seen);
  const int key_end = kv_len < max_pos + 1 ? kv_len : max_pos + 1;
  return key_end > 0 ? (key_end + kU2Keys - 1) / kU2Keys : 0;
}
// Key-range splits of a pair: as many as leave every split kU2MinSplitTiles tiles, as the batch's pairs leave pair
// slots for, and as the launch has.
__device__ __forceinline__ int u2_split_count(const Umma2Params& p, int n_tiles, int total_pairs, int launched) {
  const int room = p.pair_slots / (total_pairs * kHkv > 0 ? total_pairs * kHkv : 1);
  int splits = n_tiles >= kU2SplitFrom ? n_tiles / kU2MinSplitTiles : 1;
  splits = splits < room ? splits : room;
  splits = splits < launched ? splits : launched;
  return splits > 1 ? splits : 1;
}

__global__ void __launch_bounds__(kU2Threads, 1)
prefill_umma2_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                     const Umma2Params p) {
  extern __shared__ unsigned char u2_smem_raw[];
  Umma2Smem& sm = *reinterpret_cast<Umma2Smem*>((reinterpret_cast<uintptr_t>(u2_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.y;
  const int rank = blockIdx.x & 1;  // in the pair; 2 blockIdx.z + rank in the cluster
  NVJ_U2_PHASE(0);
  NVJ_U2_NOTE(7, 0ull);
  // The pair's barriers are set up before anything is read: this runs while the kernel in front (the append of the same
  // tokens, usually) is still at work.
  if (threadIdx.x == 32) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&k_map)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&v_map)) : "memory");
  }
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&sm.q_full), 2 * kU2SoftmaxThreads / 32);
    for (int i = 0; i < kU2Stages; ++i) {
      mbar_init(smem_u32(&sm.k_full[i]), 1);
      mbar_init(smem_u32(&sm.v_full[i]), 1);
      mbar_init(smem_u32(&sm.k_empty[i]), 1);
      mbar_init(smem_u32(&sm.v_empty[i]), 1);
    }
    mbar_init(smem_u32(&sm.s_read), kU2SoftmaxThreads / 32);  // one group of each CTA
    mbar_init(smem_u32(&sm.o_full), 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&sm.s_full[i]), 1);
      mbar_init(smem_u32(&sm.p_full[i]), kU2SoftmaxThreads / 32);
      mbar_init(smem_u32(&sm.pv_done[i][0]), 1);
      mbar_init(smem_u32(&sm.pv_done[i][1]), 1);
      for (int q = 0; q < 4; ++q) mbar_init(smem_u32(&sm.m_full[q][i]), 1);
    }
    sm.abort_flag = 0;
    mbar_fence_init();
  }
  cl_sync();  // the peer's barriers exist before anything is sent to them (this barrier covers the CTA's own threads)
  pdl_wait();
  // Tensor memory between the wait and the release (umma.cuh).  Whatever follows may take its places behind it, the decode pass of
  // a mixed batch among it (it runs beside, on the SMs this grid leaves).
  if (warp == 1) {
    tmem2_alloc(smem_u32(&sm.tmem_base), kU2TmemCols);
    if (lane == 0) {
      if (p.beside && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) st_release_gpu(p.beside, 1);
      pdl_release();
    }
  }
  auto leave = [&] {  // the whole cluster leaves without having touched its tensor memory
    cl_sync();
    if (warp == 1) tmem2_dealloc(sm.tmem_base, kU2TmemCols);
  };

  // ---- which (table row, pair of 32-token tiles) this cluster serves; every warp of its CTAs computes the same
  const U2Tile tile = u2_find_tile(p, blockIdx.x >> 1, gridDim.x >> 1, rank, gridDim.z > 1, lane);
  const int row = tile.row, tok0 = tile.tok0, ntok = tile.ntok;
  if (blockIdx.z > 0 && !tile.any_long) return leave();  // no row's key range is long enough to be split
  if (p.counted && blockIdx.x == 0 && row >= 0 && threadIdx.x == 0) atomicOr(p.status, NVJ_DEV_BAD_LENGTH);
  if (row < 0) {
    if (p.zero_fill && tile.idle == 0 && blockIdx.z == 0) {
      // the first idle cluster (there is always one) zeroes the padding tokens, a quarter per CTA of the cluster pair x KV head
      int real = p.query_start_loc[p.rows];
      real = real < p.token_bucket ? real : p.token_bucket;
      const long long n4 = (long long)(p.token_bucket - real) * kHq * kD / 4;
      float4* pad = reinterpret_cast<float4*>(p.out + (long long)real * kHq * kD);
      const int part = rank * kHkv + kvh;
      for (long long i = (long long)part * kU2Threads + threadIdx.x; i < n4; i += 2LL * kHkv * kU2Threads)
        pad[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return leave();
  }

  // What bounds the key range, the row's first 128 block ids (the producer's first eight tiles are among them, mostly, whichever split this
  // is) and the query rows are asked for together, and in this order: behind the 64 KiB of queries the few positions came 0.5 us later.
  const int seen = u2_last_positions(p, tile, rank, lane);
  int early_ids[4] = {-1, -1, -1, -1};
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i * 32 + lane < p.table_width && (i == 0 || gridDim.z > 1)) early_ids[i] = ld_in_turn(p.block_tables + (long long)row * p.table_width + i * 32 + lane);
  }
  uint4 qv[4][4];
  if (warp >= 2 && p.q_dtype == NVJ_BF16) u2_request_q(p, tok0, ntok, kvh, warp, lane, qv);
  int kv_len = tile.kv_len;
  if (kv_len > p.table_width * kBlk) {
    if (threadIdx.x == 0 && rank == 0) atomicOr(p.status, NVJ_DEV_BAD_LENGTH);
    kv_len = p.table_width * kBlk;
  }
  const int n_tiles = u2_key_tiles(seen, kv_len);
  if (n_tiles == 0) {  // same decision in both CTAs; a row without keys produces zeros
    if (p.zero_fill && blockIdx.z == 0) {
      for (int i = threadIdx.x; i < ntok * kG * (kD / 4); i += kU2Threads) {
        const int t = i / (kG * (kD / 4)), rest = i - t * (kG * (kD / 4));
        reinterpret_cast<float4*>(p.out + ((long long)(tok0 + t) * kHq + kvh * kG) * kD)[rest] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    return leave();
  }

  // Key-range splits of this pair: as many as leave every split kU2MinSplitTiles tiles and as the batch's pairs
  // leave pair slots for; the splits beyond that have nothing to do (all CTAs of the cluster decide alike).
  int splits = 1, tile0 = 0, my_tiles = n_tiles;
  if (gridDim.z > 1) {
    splits = u2_split_count(p, n_tiles, tile.total, (int)gridDim.z);
    if ((int)blockIdx.z >= splits) {
      if (splits > 1) cl_sync();  // the others' barrier in front of their fold
      return leave();
    }
    tile0 = (int)blockIdx.z * n_tiles / splits;
    my_tiles = ((int)blockIdx.z + 1) * n_tiles / splits - tile0;
  }

  int first_ids = early_ids[0];
  if (warp == 0 && tile0 > 0) {
    const int bi = tile0 * 4 + lane;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int id = __shfl_sync(0xffffffffu, early_ids[i], bi & 31);
      if (bi >> 5 == i) first_ids = id;
    }
    if (bi >= 128 && bi < p.table_width) first_ids = p.block_tables[(long long)row * p.table_width + bi];
  }
  // The tensor memory's address goes from warp 1 to the softmax warps, which have their queries on the way; the producer, which
  // needs neither, is not held up (behind a barrier of the whole CTA its first copies went out 0.6 us later).
  if (warp == 1) {
    tc_fence_before_sync();
    asm volatile("bar.arrive %0, %1;" ::"r"(6), "r"(kU2SoftmaxThreads + 32) : "memory");
  } else if (warp >= 2) {
    named_bar_sync(6, kU2SoftmaxThreads + 32);
    tc_fence_after_sync();
  }
  const uint32_t tmem = sm.tmem_base;  // (not used by warp 0)
  NVJ_U2_PHASE(1);
  NVJ_U2_NOTE(7, (unsigned long long)my_tiles);

  if (warp == 0) u2_producer(&k_map, &v_map, p, sm, row, kvh, kv_len, tile0, my_tiles, rank, lane, first_ids);
  else if (warp == 1) { if (rank == 0) u2_mma_warp(sm, p, tmem, my_tiles); }
  else u2_softmax_warps(sm, p, tmem, tok0, ntok, kvh, kv_len, tile0, my_tiles, splits, warp, lane, qv);

  tc_fence_before_sync();
  __syncthreads();
  bool odd = false;
  if (splits > 1) {
    cl_sync();  // every split's rows are staged
    odd = u2_fold_splits(sm, p, tok0, ntok, kvh, rank, splits, warp, lane);
    NVJ_U2_PHASE(5);
  }
  if (sm.abort_flag) {  // give copies and MMAs in flight time to land before memory is released
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  // CTA 0's MMAs read this CTA's shared and tensor memory until its last commit, which its softmax warps have waited for; the other splits
  // its rows.
  cl_sync_read(odd);
  NVJ_U2_PHASE(6);
  if (warp == 1) tmem2_dealloc(tmem, kU2TmemCols);
}

static int u2_pair_slots() {  // CTA pairs that run at once: half the SMs of the current device
  static PerDeviceFlags slots;
  const int dev = current_device();
  if (dev < 0) return 0;
  int n = slots.v[dev].load(std::memory_order_acquire);
  if (n == 0) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    n = sms / 2;
    slots.v[dev].store(n, std::memory_order_release);
  }
  return n;
}

constexpr int kU2SmemBytes = (int)sizeof(Umma2Smem) + 1024;
static_assert(kU2SmemBytes <= 232448, "tiles exceed the shared memory of one CTA");

// The launch of a grid of (2 x pairs, KV heads, splits) CTAs in clusters of a pair's splits, with the attributes in `attr`.
static cudaLaunchConfig_t u2_config(dim3 grid, cudaStream_t stream, cudaLaunchAttribute (&attr)[2]) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kU2Threads, 1, 1);
  cfg.dynamicSmemBytes = kU2SmemBytes;
  cfg.stream = stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = grid.z;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}
static cudaError_t u2_launch(dim3 grid, cudaStream_t stream, const CUtensorMap& k_map, const CUtensorMap& v_map, const Umma2Params& p) {
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = u2_config(grid, stream, attr);
  return cudaLaunchKernelEx(&cfg, prefill_umma2_kernel, k_map, v_map, p);
}
// Clusters of `splits` pairs that the current device holds at once (asked for once per device; 0 when it does not say).
static int u2_clusters_at_once(int splits) {
  static PerDeviceFlags known[kU2MaxSplits + 1];  // the number + 1
  const int dev = current_device();
  if (dev < 0) return 0;
  int n = known[splits].v[dev].load(std::memory_order_acquire);
  if (n == 0) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = u2_config(dim3(2 * 74, kHkv, splits), nullptr, attr);
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, prefill_umma2_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      clusters = 0;
    }
    n = clusters + 1;
    known[splits].v[dev].store(n, std::memory_order_release);
  }
  return n - 1;
}

// Whether launch_prefill_umma2 will take a batch with these parameters (a caller that knows so need not zero the output).
bool prefill_umma2_usable(float scale, long long num_blocks) { return scale > 0.f && num_blocks >= 1 && tensor_maps_available(); }

// Returns NVJ_ERR_UNSUPPORTED when the driver offers no tensor-map encoder or the scale is not positive.
int launch_prefill_umma2(const void* q, int q_dtype, const char* k_cache, const char* v_cache,
                         long long num_blocks, const int32_t* block_tables, int table_width,
                         const int32_t* kv_lens, const int32_t* positions, const int32_t* query_start_loc,
                         int rows, int token_bucket, float scale, float* out, int32_t* status,
                         int skip_single, int split_p, int tile_pairs, bool may_split, int32_t* beside, cudaStream_t stream) {
  static PerDeviceFlags opted_in;
  if (!(scale > 0.f) || num_blocks < 1 || !tensor_maps_available()) return NVJ_ERR_UNSUPPORTED;
  if (!once_per_device(opted_in, [](int) {
        return cudaFuncSetAttribute(prefill_umma2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kU2SmemBytes) == cudaSuccess;
      }))
    return NVJ_ERR_LAUNCH;
  CUtensorMap k_map, v_map;
  if (!grouped_map_cached(&k_map, k_cache, (uint64_t)num_blocks * kBlk, 4) ||
      !grouped_map_cached(&v_map, v_cache, (uint64_t)num_blocks * kBlk, 2))
    return NVJ_ERR_UNSUPPORTED;
  // The kernel zeroes what no tile writes itself (padding tokens, rows of several tokens without keys), and the
  // decode-row pass of a mixed batch does the same for its rows: no memset launch in front of a batch.
  Umma2Params p{};
  p.zero_fill = 1;
  p.q = q; p.q_dtype = q_dtype;
  p.block_tables = block_tables; p.kv_lens = kv_lens; p.positions = positions; p.query_start_loc = query_start_loc;
  p.out = out; p.status = status; p.num_blocks = num_blocks; p.rows = rows; p.token_bucket = token_bucket;
  p.table_width = table_width; p.skip_single = skip_single; p.scale = scale; p.split_p = split_p;
  p.beside = beside;
  // Clusters: one per pair of tiles and one that stays idle (it zeroes the padding).  Without the caller's count, at most
  // so many; the ones too many cost a batch of many rows and few tiles its start (34 rows, 8 pairs: 43 clusters per head,
  // two waves of CTAs that only set themselves up and leave).
  const int most_pairs = (token_bucket + 2 * kU2Tokens - 1) / (2 * kU2Tokens) + rows;
  const int pairs = tile_pairs >= 0 && tile_pairs + 1 < most_pairs ? tile_pairs + 1 : most_pairs;
  p.counted = pairs < most_pairs;
  // Key-range splits: only while the batch leaves pair slots free, by the most pairs that it can hold (a batch of many short rows
  // is launched whole: its extra splits would only scan the rows and leave, 200 us on 256 rows of 4 tokens); the kernel settles
  // the number per pair from what the batch really holds.  The pairs of a tile are one cluster, and a GPC has room for whole ones only.
  int splits = 1;
  if (may_split) {
    p.pair_slots = u2_pair_slots();
    for (int s = 2; s <= kU2MaxSplits && s * pairs * kHkv <= p.pair_slots; ++s)
      if ((pairs - 1) * kHkv <= u2_clusters_at_once(s)) splits = s;  // (one pair per head, if not more, is idle and leaves at once)
  }
  return u2_launch(dim3(2 * pairs, kHkv, splits), stream, k_map, v_map, p) == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

}  // namespace nvj

#ifdef NVJ_PHASE_TIMING
extern "C" int nvj_debug_prefill_phase_ns(unsigned long long* host_out) {  // [512][8]
  return cudaMemcpyFromSymbol(host_out, nvj::g_u2_phase_ns, sizeof(nvj::g_u2_phase_ns)) == cudaSuccess ? 0 : 1;
}
#endif
