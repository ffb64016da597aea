// Paged GQA decode attention for rows of 9 - 16 query tokens on the 5th-generation tensor cores, on ranges: the form of
// paged_decode_umma.cu (which has the work split, the semantics and the launch) with the query rows as the rows of the tile.
//
// The 36 - 64 query rows of one KV head sit in lanes 0..63 of a 128-row UMMA tile (the other lanes compute on whatever they hold and
// are never read): per tile of 64 keys and KV head 16 MMAs of N = 64 for the scores and eight of N = 256 for the weighted sum, ~1500 tensor
// cycles against ~3000 cycles of HBM time.  Ahead of the transposed form here because its tiles are smaller and its ring is deeper
// (64 columns leave room for two 64 KiB slots): 64 rows of 9 tokens under 64 blocks 34.7 us, transposed 40.8; 128 under 40 43.8 and 51.0.
//
// A range belongs to a pair of CTAs, one per KV head.  Keys are walked in tiles of up to four blocks
// that never straddle a row; a block's K lands as [8-key group][64-d chunk][8 keys][128 B] (the groups of a tile are then evenly
// spaced and the whole tile is one N = 64 operand), its V as [chunk][16 keys][128 B] (P V contracts 16 keys per MMA), one 8 KiB
// TMA box each.  One CTA per SM (192 KiB of shared memory: three tiles of K and of V in flight; 512 TMEM columns: query rows,
// scores, weights, output).
//   warps 0, 1  (a warp may only touch the 32 TMEM lanes of its quarter)
//            softmax: lane r = query row r = token * 4 + head of the group.  Per tile it reads the scores (tcgen05.ld), which frees
//            them for the next tile's, masks, keeps the running maximum lazily (O in tensor memory is rescaled only when a tile exceeds
//            it by 2^8) and writes the weights as two bf16 terms (hi + lo).  At the end of a row segment it reads half of O's columns.
//   warps 4, 5  on the same lanes: the other half of O, and the next segment's query rows into tensor memory as soon as the
//            segment's last scores have been computed.
//   warp 2   MMA issue: S(t + 1) = Q K(t + 1)^T while the softmax is at work on S(t), then O += P(t) V(t) once the weights are
//            written.  tcgen05.commit releases ring stages and signals the other warps.
//   warp 3   K producer, warp 7 V producer: block ids straight from the block table (32 at a time), TMA boxes into the rings.

#include <cuda.h>

#include "decode_parts.cuh"
#include "umma.cuh"

namespace nvj {
namespace query_rows {

constexpr int kUdStages = 3;      // tiles (K and V of one KV head for up to 64 keys: 64 KiB) in flight
constexpr int kUdTileBlocks = 4;  // blocks per tile: 64 keys
constexpr int kUdAheadBlocks = 28;  // prefetched ahead of the wait, as in paged_decode_umma.cu
constexpr int kUdTmemCols = 512;
constexpr int kUdColQ = 0;        // query rows as the A operand: 256 bf16 per row = 128 columns
constexpr int kUdColS = 128;      // scores of a tile
constexpr int kUdColP = 192;      // its weights: hi 32 columns, lo 32
constexpr int kUdColO = 256;      // output accumulator: columns [256, 512)
constexpr int kUdHalfBlock = kBlk * kD * 2;  // K (or V) of one KV head of one block: 8 KiB
constexpr float kUdRescaleGap = 8.f;

struct UdSmem {
  alignas(1024) char k[kUdStages][kUdTileBlocks][kUdHalfBlock];    // [stage][block][8-key group][64-d chunk][8 keys][128 B], swizzled
  alignas(1024) char v[kUdStages][kUdTileBlocks][kUdHalfBlock];    // [stage][block][64-d chunk][16 keys][128 B], swizzled
  alignas(8) unsigned long long k_full[kUdStages], k_empty[kUdStages], v_full[kUdStages], v_empty[kUdStages],
      q_full, q_free, s_full, s_read, p_full, pv_done, o_ready[2], o_free;
  float inv[64];  // per query row: what the segment's output is scaled by
  int scan[16];
  int start_b, start_j, abort_flag, begun;
  uint32_t tmem_base;
};

// Position in a ring of kUdStages.
struct UdRing {
  int at = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void step() {
    if (++at == kUdStages) { at = 0; phase ^= 1u; }
  }
};
// ---- warps 3 and 7: TMA loads of K and of V --------------------------------------------------------------
// The first round of stages is all the K warp's, in the order in which the tiles want it (with both warps at it, the first tile's K
// would share the SM's intake with its V).
template <bool kK>
__device__ __forceinline__ void ud_producer(const CUtensorMap* k_map, const CUtensorMap* v_map, const DecodeParams& p, UdSmem& sm, int kvh,
                                            int b, int j, long long g, long long g1, int lane) {
  const int oob = (int)(p.num_blocks * kBlk);  // a box that starts here is filled with zeros
  uint64_t policy;  // every block is read once: do not let it displace what the L2 is good for
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  Seg s;
  UdRing at;
  bool reuse = false;  // the stage has been used before
  while (next_seg(p, b, j, g, g1, s)) {
    const long long tbase = decode_table_base(p, s.b);
    for (int jb = s.j0; jb < s.j1; jb += 32) {  // 32 block ids = 8 tiles at a time
      const int n = s.j1 - jb < 32 ? s.j1 - jb : 32;
      int id = -1;
      if (lane < n) {
        id = p.block_tables[tbase + jb + lane];
        if (id < 0 || id >= p.num_blocks) {
          atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
          id = -1;
        }
      }
      for (int i0 = 0; i0 < n; i0 += kUdTileBlocks) {
        const int cnt = n - i0 < kUdTileBlocks ? n - i0 : kUdTileBlocks;
        if (reuse && !um_wait(kK ? &sm.k_empty[at.at] : &sm.v_empty[at.at], at.phase ^ 1u, &sm.abort_flag, p.status)) return;
        const int blk = __shfl_sync(kFullMask, id, i0 + (lane & (kUdTileBlocks - 1)));
        const int token = blk >= 0 ? blk * kBlk : oob;
        if (kK) {
          const uint32_t full = smem_u32(&sm.k_full[at.at]);
          if (lane == 0) mbar_arrive_expect_tx(full, (uint32_t)cnt * kUdHalfBlock);
          __syncwarp();
          if (lane < cnt) tma_load_k_half(smem_u32(&sm.k[at.at][lane][0]), k_map, token / 8, kvh, full, policy);  // a lane per block
        }
        if (kK != reuse) {
          const uint32_t full = smem_u32(&sm.v_full[at.at]);
          if (lane == 0) mbar_arrive_expect_tx(full, (uint32_t)cnt * kUdHalfBlock);
          __syncwarp();
          if (lane < cnt) tma_load_v_half(smem_u32(&sm.v[at.at][lane][0]), v_map, token, kvh, full, policy);
        }
        __syncwarp();
        at.step();
        if (at.at == 0) reuse = true;
      }
    }
  }
}

// ---- warp 2: MMA issue --------------------------------------------------------------------------
// Walks the range's tiles: once for the scores, once for the weighted sums.
struct UdTiles {
  Seg s;
  int b, j, t, nt, seg;  // tile t of the segment's nt; segments so far
  long long g;
  UdRing at;
  bool have;
  __device__ __forceinline__ void enter(const DecodeParams& p, long long g1) {
    have = next_seg(p, b, j, g, g1, s);
    t = 0;
    nt = have ? (s.j1 - s.j0 + kUdTileBlocks - 1) / kUdTileBlocks : 0;
  }
  __device__ __forceinline__ void step(const DecodeParams& p, long long g1) {
    at.step();
    if (++t == nt) { ++seg; enter(p, g1); }
  }
};

__device__ __forceinline__ void ud_mma_warp(UdSmem& sm, const DecodeParams& p, uint32_t tmem, int b, int j, long long g,
                                            long long g1) {
  const uint64_t k_desc0 = umma_desc(smem_u32(&sm.k[0][0][0]), 16, 4 * 8 * 128);   // K: keys are rows (groups of 8: 4 KiB apart), dims contracted
  const uint64_t v_desc0 = umma_desc(smem_u32(&sm.v[0][0][0]), kBlk * 128, 1024);  // V: 64-d chunks 2 KiB apart, keys contracted
  UdTiles sc{};  // the next scores to be issued
  sc.b = b; sc.j = j; sc.g = g;
  sc.enter(p, g1);
  UdTiles pv = sc;  // the next weighted sum
  uint32_t scored = 0, done = 0;  // tiles so far
  // Scores of the next tile (columns of blocks that the tile does not have are computed from whatever the stage holds there and
  // masked by the softmax warp), once the softmax has read the scores before.
  auto issue_scores = [&] {
    if (sc.t == 0 && !um_wait(&sm.q_full, (uint32_t)sc.seg & 1u, &sm.abort_flag, p.status)) return false;
    if (!um_wait(&sm.k_full[sc.at.at], sc.at.phase, &sm.abort_flag, p.status)) return false;
    if (scored > 0 && !um_wait(&sm.s_read, (scored - 1) & 1u, &sm.abort_flag, p.status)) return false;
    tc_fence_after_sync();
    if (um_elect_one()) {
      constexpr uint32_t idesc = umma_idesc(kUdTileBlocks * kBlk, false);
      const uint64_t k_desc = k_desc0 + (uint64_t)((sc.at.at * kUdTileBlocks * kUdHalfBlock) >> 4);
#pragma unroll
      for (int ks = 0; ks < 16; ++ks)  // 16 dims per MMA: 8 columns of Q; K chunk ks / 4, 32 bytes into its swizzled rows
        umma_bf16_ts(tmem + kUdColS, tmem + kUdColQ + ks * 8, k_desc + (uint64_t)(((ks >> 2) * (8 * 128) + (ks & 3) * 32) >> 4), idesc,
                     ks > 0 ? 1u : 0u);
      umma_commit(smem_u32(&sm.s_full));
      umma_commit(smem_u32(&sm.k_empty[sc.at.at]));
      if (sc.t == sc.nt - 1) umma_commit(smem_u32(&sm.q_free));
    }
    __syncwarp();
    sc.step(p, g1);
    ++scored;
    return true;
  };
  while (pv.have) {
    if (scored == done && !issue_scores()) return;
    // The next tile's scores go first, unless they would have to wait for keys or queries; those of the first tiles, whose keys have
    // been on their way from the start, in any case.  (Looking at both barriers in turn until one is ready takes more from the other
    // warps than it gives: 66.0 -> 68.5 us.)
    if (sc.have && scored == done + 1 &&
        (scored < kUdStages || (um_test(&sm.k_full[sc.at.at], sc.at.phase) && (sc.t > 0 || um_test(&sm.q_full, (uint32_t)sc.seg & 1u)))) &&
        !issue_scores())
      return;
    if (!um_wait(&sm.v_full[pv.at.at], pv.at.phase, &sm.abort_flag, p.status)) return;
    if (!um_wait(&sm.p_full, done & 1u, &sm.abort_flag, p.status)) return;
    // the first P V of a segment overwrites O: the segment before must have been read out
    if (pv.t == 0 && pv.seg > 0 && !um_wait(&sm.o_free, (uint32_t)(pv.seg - 1) & 1u, &sm.abort_flag, p.status)) return;
    tc_fence_after_sync();
    if (um_elect_one()) {
      constexpr uint32_t idesc = umma_idesc(kD, true);
      const int nblk = pv.s.j1 - pv.s.j0, cnt = nblk - pv.t * kUdTileBlocks < kUdTileBlocks ? nblk - pv.t * kUdTileBlocks : kUdTileBlocks;
      for (int i = 0; i < cnt; ++i) {  // 16 keys per MMA: 8 columns of P, the block's two 8-key groups of V
        const uint64_t dv = v_desc0 + (uint64_t)(((pv.at.at * kUdTileBlocks + i) * kUdHalfBlock) >> 4);
        umma_bf16_ts(tmem + kUdColO, tmem + kUdColP + i * 8, dv, idesc, (pv.t > 0 || i > 0) ? 1u : 0u);
        umma_bf16_ts(tmem + kUdColO, tmem + kUdColP + 32 + i * 8, dv, idesc, 1u);
      }
      umma_commit(smem_u32(&sm.v_empty[pv.at.at]));
      umma_commit(smem_u32(&sm.pv_done));
    }
    __syncwarp();
    ++done;
    pv.step(p, g1);
  }
}

// A segment's output out of tensor memory, columns [128 half, 128 half + 128): the row, or the range's partial.
__device__ __forceinline__ void ud_store_output(const UdSmem& sm, const DecodeParams& p, uint32_t tmem, const Seg& s, int kvh, int range, int row,
                                                int half) {
  const int tok = row >> 2, head = row & 3;
  const bool whole_row = (s.j0 == 0 && s.j1 == s.nb);
  const int slot = partial_slot(range, s.j0 == 0);
  const float inv = sm.inv[row];
  const long long at = whole_row ? ((long long)s.b * p.width + tok) * kHq + kvh * kG + head
                                 : (long long)slot * (p.width * kHq) + tok * kHq + kvh * kG + head;
  float* dst = (whole_row ? p.out : p.part_acc) + at * kD + half * (kD / 2);
#pragma unroll 1
  for (int cc = 0; cc < kD / 64; ++cc) {
    float o[32];
    tmem_ld32(tmem + kUdColO + half * (kD / 2) + cc * 32, o);
    if (tok < p.width) {
#pragma unroll
      for (int i = 0; i < 32; i += 4)
        *reinterpret_cast<float4*>(dst + cc * 32 + i) = make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
    }
  }
}

// ---- warps 0 and 1: softmax, half of the output ------------------------------------------------------------
__device__ __forceinline__ void ud_softmax_warp(UdSmem& sm, const DecodeParams& p, uint32_t tmem, int kvh, int b, int j,
                                                long long g, long long g1, int range, int row) {
  const int tok = row >> 2, head = row & 3;
  const bool real = tok < p.width;
  const float scale_log2 = p.scale * kLog2e;
  Seg s;
  UdRing at;
  uint32_t done = 0;  // tiles so far
  while (next_seg(p, b, j, g, g1, s)) {
    const int my_pos = real ? (p.positions ? p.positions[(long long)s.b * p.width + tok] : 0x7fffffff) : -1;
    const int last_key = my_pos < s.len - 1 ? my_pos : s.len - 1;  // last key this row may see
    float m_row = -INFINITY, l_row = 0.f;                           // m_row in units of log2(e) * scale
    const int nblk = s.j1 - s.j0, nt = (nblk + kUdTileBlocks - 1) / kUdTileBlocks;
    for (int t = 0; t < nt; ++t, ++done, at.step()) {
      if (!um_wait(&sm.s_full, done & 1u, &sm.abort_flag, p.status)) return;
      tc_fence_after_sync();
      float sc[64];
      {
        float a[32];
        tmem_ld32(tmem + kUdColS, a);
#pragma unroll
        for (int i = 0; i < 32; ++i) sc[i] = a[i];
        tmem_ld32(tmem + kUdColS + 32, a);
#pragma unroll
        for (int i = 0; i < 32; ++i) sc[32 + i] = a[i];
      }
      tc_fence_before_sync();
      mbar_arrive(smem_u32(&sm.s_read));
      const int cnt = nblk - t * kUdTileBlocks < kUdTileBlocks ? nblk - t * kUdTileBlocks : kUdTileBlocks;
      int lim = last_key - (s.j0 + t * kUdTileBlocks) * kBlk;  // columns [0, lim] are visible
      lim = lim < cnt * kBlk - 1 ? lim : cnt * kBlk - 1;       // columns of blocks the tile does not have hold old scores
      float tmax = -INFINITY;
#pragma unroll
      for (int i = 0; i < 64; ++i) {
        sc[i] = i <= lim ? sc[i] : -INFINITY;
        tmax = fmaxf(tmax, sc[i]);
      }
      tmax *= scale_log2;  // scale > 0
      if (t == 0) {
        m_row = tmax;
      } else if (__any_sync(kFullMask, tmax > m_row + kUdRescaleGap)) {
        // rare: raise the maxima and rescale O, once the last P V has landed
        if (!um_wait(&sm.pv_done, (done - 1) & 1u, &sm.abort_flag, p.status)) return;
        tc_fence_after_sync();
        const float m_new = fmaxf(m_row, tmax);
        const float f = m_new == -INFINITY ? 1.f : ex2_approx(m_row - m_new);
        m_row = m_new;
        l_row *= f;
#pragma unroll 1
        for (int cc = 0; cc < kD / 32; ++cc) {
          float o[32];
          tmem_ld32(tmem + kUdColO + cc * 32, o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] *= f;
          tmem_st32(tmem + kUdColO + cc * 32, o);
        }
      }
      const float neg_m = m_row == -INFINITY ? 0.f : -m_row;
      uint32_t hi[32], lo[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        const float p0 = ex2_approx(fmaf(sc[2 * e], scale_log2, neg_m)), p1 = ex2_approx(fmaf(sc[2 * e + 1], scale_log2, neg_m));
        l_row += p0 + p1;
        const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
        const __nv_bfloat162 r2 = __floats2bfloat162_rn(p0 - __low2float(h), p1 - __high2float(h));
        hi[e] = *reinterpret_cast<const uint32_t*>(&h);
        lo[e] = *reinterpret_cast<const uint32_t*>(&r2);
      }
      // P V of the tile before has read its weights (every phase of pv_done is observed in turn: a parity wait tells only two
      // consecutive phases apart)
      if (done >= 1 && !um_wait(&sm.pv_done, (done - 1) & 1u, &sm.abort_flag, p.status)) return;
      {  // P(t) as the A operand of P V: keys 2j, 2j + 1 in column j; hi in columns [0, 32), lo in [32, 64)
        uint32_t w[16];
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
#pragma unroll
          for (int i = 0; i < 16; ++i) w[i] = q4 < 2 ? hi[(q4 & 1) * 16 + i] : lo[(q4 & 1) * 16 + i];
          tmem_st16(tmem + kUdColP + q4 * 16, w);
        }
      }
      tmem_st_wait();
      if (t == nt - 1 && s.j1 == s.nb && (s.len & (kBlk - 1))) {
        // V rows of the last block behind the last key weigh nothing, but may hold anything: 0 x infinity is not 0.  The 64 threads of
        // the two warps are the block's 4 chunks x 16 keys.
        if (!um_wait(&sm.v_full[at.at], at.phase, &sm.abort_flag, p.status)) return;
        if ((row & (kBlk - 1)) >= (s.len & (kBlk - 1))) {
          char* rest = &sm.v[at.at][cnt - 1][row * 128];
#pragma unroll
          for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(rest + i * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async_smem();
      }
      tc_fence_before_sync();
      mbar_arrive(smem_u32(&sm.p_full));
    }
    // ---- end of the segment: half of O for the warp that helps, half here
    if (!um_wait(&sm.pv_done, (done - 1) & 1u, &sm.abort_flag, p.status)) return;
    tc_fence_after_sync();
    const bool whole_row = (s.j0 == 0 && s.j1 == s.nb);
    sm.inv[row] = whole_row ? (l_row > 0.f ? 1.f / l_row : 0.f) : 1.f;
    tc_fence_before_sync();
    mbar_arrive(smem_u32(&sm.o_ready[row >> 5]));
    ud_store_output(sm, p, tmem, s, kvh, range, row, 0);
    if (real && !whole_row)
      *reinterpret_cast<float2*>(p.part_ml + ((long long)partial_slot(range, s.j0 == 0) * (p.width * kHq) + tok * kHq + kvh * kG + head) * 2) =
          make_float2(m_row == -INFINITY ? kNegBig : m_row, l_row);
    tc_fence_before_sync();  // the next segment's first P V overwrites what was just read
    mbar_arrive(smem_u32(&sm.o_free));
  }
}

// ---- warps 4 and 5: query rows, the other half of the output -----------------------------------------------
// Query row `row` of table row `row_b` into tensor memory: 256 dims -> 128 columns, two bf16 per column; sixteen 16-byte loads in
// flight at a time (one at a time, the eight round trips to memory cost a segment more than its epilogue), the first sixteen
// before the wait for the columns.  `n`: segments staged before.
__device__ __forceinline__ bool ud_stage_q(UdSmem& sm, const DecodeParams& p, uint32_t tmem, int kvh, int row_b, int row, uint32_t n) {
  const int tok = row >> 2, head = row & 3;
  const bool real = tok < p.width;
  const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.q) +
                                                    (((long long)row_b * p.width + (real ? tok : 0)) * kHq + kvh * kG + head) * kD);
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    uint4 u[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) u[i] = real ? ld_stream_u4(src + half * 16 + i) : make_uint4(0u, 0u, 0u, 0u);
    if (half == 0 && n > 0) {  // the last scores of the segment before have been computed
      if (!um_wait(&sm.q_free, (n - 1) & 1u, &sm.abort_flag, p.status)) return false;
      tc_fence_after_sync();
    }
#pragma unroll
    for (int part = 0; part < 4; ++part) {  // 32 dims = 16 columns at a time
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        w[4 * i] = u[part * 4 + i].x; w[4 * i + 1] = u[part * 4 + i].y; w[4 * i + 2] = u[part * 4 + i].z; w[4 * i + 3] = u[part * 4 + i].w;
      }
      tmem_st16(tmem + kUdColQ + half * 64 + part * 16, w);
    }
  }
  tmem_st_wait();
  tc_fence_before_sync();
  mbar_arrive(smem_u32(&sm.q_full));
  return true;
}

__device__ __forceinline__ void ud_helper_warp(UdSmem& sm, const DecodeParams& p, uint32_t tmem, int kvh, int b, int j, long long g,
                                               long long g1, int range, int row) {
  Seg s, nxt;
  bool have = next_seg(p, b, j, g, g1, s);
  if (have && !ud_stage_q(sm, p, tmem, kvh, s.b, row, 0)) return;
  for (uint32_t n = 0; have; ++n) {
    const bool more = next_seg(p, b, j, g, g1, nxt);
    if (more && !ud_stage_q(sm, p, tmem, kvh, nxt.b, row, n + 1)) return;
    if (!um_wait(&sm.o_ready[row >> 5], n & 1u, &sm.abort_flag, p.status)) return;
    tc_fence_after_sync();
    ud_store_output(sm, p, tmem, s, kvh, range, row, 1);
    tc_fence_before_sync();
    mbar_arrive(smem_u32(&sm.o_free));
    s = nxt;
    have = more;
  }
}

// A CTA of the launch that folds the partials fits beside this one and waits in place.
__global__ void __maxnreg__(kUmmaQueryRowsRegs)
decode_umma_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, DecodeParams p) {
  extern __shared__ unsigned char ud_smem_raw[];
  UdSmem& sm = *reinterpret_cast<UdSmem*>((reinterpret_cast<uintptr_t>(ud_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = blockIdx.x & 1, range = blockIdx.x >> 1, ranges = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&k_map)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&v_map)) : "memory");
    sm.start_b = p.batch; sm.start_j = 0; sm.abort_flag = 0; sm.begun = 0;
    for (int i = 0; i < kUdStages; ++i) {
      mbar_init(smem_u32(&sm.k_full[i]), 1);
      mbar_init(smem_u32(&sm.k_empty[i]), 1);
      mbar_init(smem_u32(&sm.v_full[i]), 1);
      mbar_init(smem_u32(&sm.v_empty[i]), 1);
    }
    constexpr uint32_t quarters = 2;  // of the TMEM lanes: 32 query rows each
    mbar_init(smem_u32(&sm.q_full), 32 * quarters);
    mbar_init(smem_u32(&sm.q_free), 1);
    mbar_init(smem_u32(&sm.s_full), 1);
    mbar_init(smem_u32(&sm.s_read), 32 * quarters);
    mbar_init(smem_u32(&sm.o_ready[0]), 32);
    mbar_init(smem_u32(&sm.o_ready[1]), 32);
    mbar_init(smem_u32(&sm.p_full), 32 * quarters);
    mbar_init(smem_u32(&sm.pv_done), 1);
    mbar_init(smem_u32(&sm.o_free), 64 * quarters);
    mbar_fence_init();
  }
  __syncthreads();
  if (warp == 7 && p.early_ctas > 0) prefetch_ahead(p, range, ranges, kUdAheadBlocks, kvh == 0, kvh == 1, &sm.begun, lane);
  pdl_wait();
  if (threadIdx.x == 0) *static_cast<volatile int*>(&sm.begun) = 1;
  // this CTA's share of the block tables into the L2, while the lengths are on their way
  {
    const long long lines = ((long long)p.batch * p.table_width * (long long)sizeof(int32_t) + 127) / 128;
    const long long line = (long long)blockIdx.x * kDecodeThreads + threadIdx.x;
    if (line < lines) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p.block_tables) + line * 128));
  }
  // ---- pass 1: total number of blocks; zero the output of inactive rows
  int mine = 0, first_n = 0;
  for (int base = 0; base < p.batch; base += kDecodeThreads) {
    const int b = base + threadIdx.x;
    int len = 0;
    if (b < p.batch) len = decode_row_len(p, b);
    if (base == 0) first_n = blocks_in_sequence(p, (len + kBlk - 1) / kBlk);
    mine += blocks_in_sequence(p, (len + kBlk - 1) / kBlk);
    const unsigned idle = __ballot_sync(kFullMask, b < p.batch && len <= 0 && (b % (int)gridDim.x) == (int)blockIdx.x);
    for (unsigned m = idle; m; m &= m - 1) {
      const int bb = base + (warp << 5) + (__ffs(m) - 1);
      float4* o = reinterpret_cast<float4*>(p.out + (long long)bb * p.width * kHq * kD);
      for (int i = lane; i < p.width * kHq * kD / 4; i += 32) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  int total = 0;
  const int incl = cta_inclusive_scan(mine, sm.scan, total);
  if (total == 0) {
    if (kvh == 0 && threadIdx.x == 0) umma_cuts(p, ranges)[range] = kNoCut;
    return;
  }
  const Partition pt = make_partition(total, ranges);
  const long long g0 = pt.start(range);
  const long long g1 = pt.start(range + 1);
  if (range >= pt.n || g0 == g1) {
    if (kvh == 0 && threadIdx.x == 0) umma_cuts(p, ranges)[range] = kNoCut;
    return;
  }

  // ---- pass 2: locate (row, block) of g0
  long long carry = 0;
  if (p.batch <= kDecodeThreads) {  // one row per thread: the scan of pass 1 has the answer already
    const long long excl = incl - first_n;
    if (first_n > 0 && excl <= g0 && g0 < excl + first_n) { sm.start_b = threadIdx.x; sm.start_j = (int)(g0 - excl); }
    carry = g0 + 1;  // skips the loop below
  }
  for (int base = 0; base < p.batch && carry <= g0; base += kDecodeThreads) {
    const int b = base + threadIdx.x;
    int n = 0;
    if (b < p.batch) n = blocks_in_sequence(p, (decode_row_len(p, b) + kBlk - 1) / kBlk);
    int chunk_total = 0;
    const long long excl = carry + cta_inclusive_scan(n, sm.scan, chunk_total) - n;
    if (n > 0 && excl <= g0 && g0 < excl + n) { sm.start_b = b; sm.start_j = (int)(g0 - excl); }
    carry += chunk_total;
  }
  if (warp == 2) {  // tensor memory between the wait and the release (umma.cuh)
    tmem_alloc(smem_u32(&sm.tmem_base), kUdTmemCols);
    if (lane == 0) pdl_release();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sm.tmem_base;
  const int b0 = sm.start_b, j0 = sm.start_j;
  // (by a thread that has nothing to do until the first keys are there)
  if (kvh == 0 && threadIdx.x == 2 * 32) umma_cuts(p, ranges)[range] = umma_cut(p, pt, range, b0, j0, g0);

  const int quarter = warp & 3;  // of the TMEM lanes that this warp may touch: rows 32 * quarter ..
  const uint32_t mine_tmem = tmem + ((uint32_t)(quarter * 32) << 16);
  if (warp == 2) ud_mma_warp(sm, p, tmem, b0, j0, g0, g1);
  else if (warp == 3) ud_producer<true>(&k_map, &v_map, p, sm, kvh, b0, j0, g0, g1, lane);
  else if (warp == 7) ud_producer<false>(&k_map, &v_map, p, sm, kvh, b0, j0, g0, g1, lane);
  else if (quarter < 2) {
    if (warp < 4) ud_softmax_warp(sm, p, mine_tmem, kvh, b0, j0, g0, g1, range, quarter * 32 + lane);
    else ud_helper_warp(sm, p, mine_tmem, kvh, b0, j0, g0, g1, range, quarter * 32 + lane);
  }

  tc_fence_before_sync();
  __syncthreads();
  if (sm.abort_flag) {  // give copies and MMAs in flight time to land before the CTA's memory is released
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 2) tmem_dealloc(tmem, kUdTmemCols);
}

}  // namespace query_rows

// p as launch_decode_umma has it, more than 8 tokens per row.
int launch_decode_umma_query_rows(const DecodeParams& p, int ranges, const CUtensorMap& k_map, const CUtensorMap& v_map, cudaStream_t stream) {
  using namespace query_rows;
  static PerDeviceFlags smem_opted_in;
  constexpr int kSmemBytes = (int)sizeof(UdSmem) + 1024;
  static_assert(kSmemBytes <= 232448, "the tile ring exceeds the shared memory of one CTA");
  if (!once_per_device(smem_opted_in, [](int) {
        return cudaFuncSetAttribute(decode_umma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) == cudaSuccess;
      }))
    return NVJ_ERR_LAUNCH;
  launch_after(decode_umma_kernel, 2 * ranges, kDecodeThreads, kSmemBytes, stream, k_map, v_map, p);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

}  // namespace nvj
