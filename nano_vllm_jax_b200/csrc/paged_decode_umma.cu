// Paged GQA decode attention for rows of several query tokens (speculative verification, widths up to 16) on the
// 5th-generation tensor cores: tcgen05.mma with the scores and the output accumulators in tensor memory.
//
// The 4 x width query rows of a KV head are far fewer than the 128 rows of a UMMA tile, so both products are taken transposed, with
// the keys and then the dims as the tile's rows and the query rows in its columns:
//   S^T = K Q^T    [128 keys x kN], 16 MMAs over the dims, K and Q straight from shared memory;
//   O^T = V^T P^T  [2 x 128 dims x 2 kN], 16 keys per MMA: the weights enter as two bf16 terms (hi + lo) in columns of their own, added
//                  when the output is read.
// A tile of 128 keys takes 1024 tensor cycles (what reading K and V from shared memory takes) where the query rows as the tile's rows
// took 3000, most of them for lanes without a row; 64 rows of 5 tokens over 1024 - 4096 keys then ran at the board's power limit, 80 us,
// and now take 64 (append, this and the fold; 52 at the copy rate).  kN = 32 for up to 8 tokens: three accumulators take the tiles
// in turn, so that a sum is a third as long (error against 64 bits 4.4e-6 -> 2.5e-6 there).  More than 8 tokens: 64 columns,
// on clusters only; on ranges the query rows stay the tile's rows (paged_decode_umma_query_rows.cu), 64 columns and two slots are no faster.
//
// Work split.  A CTA serves one KV head: CTA pairs (ranges) or clusters (kCluster).
//   Ranges: the blocks of all rows form one sequence cut into equal ranges as in the other decode kernels (decode_parts.cuh), CTA
//   2c + h streams head h's half of every block of range c.  Rows cut over ranges are folded by a second launch.
//   Clusters, where they find a place all at once and a CTA's share is short (umma_cluster): one per (row, KV head), CTA r takes blocks r,
//   r + C, ... .  No scan in front and no fold behind: the block ids are requested together with the length and the CTAs' sums
//   meet in distributed shared memory.  2 rows of 5 tokens under 256 blocks 18.4 -> 11.7 us, 16 under 128 22.3 -> 17.3, 64 under 32 24.6 -> 18.0.
//   warps 0 - 3  softmax, thread = key: reads its scores (tcgen05.ld), masks (key < length, key <= the token's position), writes the
//                weights' terms into shared memory.  Maxima are kept lazily: the four warps vote whether a score exceeds its maximum
//                by 2^8, and only then (and in a segment's first tile) reduce the tile's maxima and rescale O in tensor memory.  At the
//                end of a row segment thread = dim: the row (whole row in this CTA), the partial with its (max, sum), or the sums for the cluster.
//   warp 4       MMA issue.
//   warp 5       TMA producer: block ids straight from the block table (32 at a time, the next row's in advance), 8 KiB boxes into a ring of
//                64 KiB slots that K and V of a tile take in turn.  (K in one slot of its own and V in half slots, the same 192 KiB: 72 us
//                instead of 68; K's next request then waits for its scores.)
//   warps 6, 7   the next segment's query rows, as soon as the segment's last scores have been computed.
// Every wait is bounded; on a timeout the kernel flags NVJ_DEV_TIMEOUT, stops issuing, lets copies in flight land
// and still frees its tensor memory.  A block id outside the pool is flagged and its box is fetched from beyond the
// tensor (zeros), so nothing foreign is read; the row's result is then meaningless but finite.
// Semantics: nanovllm_jax/kv_cache.py:852-998 with query width > 1 (key p of row b is visible to token t when
// p < seq_lens[b] and, with positions given, p <= positions[b, t]).

#include <cuda.h>

#include "decode_cluster.cuh"
#include "umma.cuh"

namespace nvj {

constexpr int kUdTileBlocks = 8;  // blocks per tile: 128 keys, the rows of a UMMA tile
constexpr int kUdTmemCols = 512;
constexpr int kUdHalfBlock = kBlk * kD * 2;                 // K (or V) of one KV head of one block: 8 KiB
constexpr int kUdSlotBytes = kUdTileBlocks * kUdHalfBlock;  // of one tile: 64 KiB
constexpr float kUdRescaleGap = 8.f;
// Blocks of a range that are prefetched ahead of the wait, while the append in front is at work (prefetch_ahead): 64 rows of 5 tokens over 1024 -
// 4096 keys 66.4 us without, 64.8 with 8, 64.8 with 16, 64.0 with 28; 128 over 2000 - 4000 135.8, 132.6, 131.4, 130.9.
constexpr int kUdAheadBlocks = 28;
constexpr int kUdMaxWidth = 16;   // 64 query rows per KV head
constexpr int kUdMaxCluster = 16;
// What a row end costs a CTA here, in blocks: 256 rows of 5 tokens under 40 blocks 57.7 us with 3, 54.9 with 6, 52.2 with 9, 51.9 with 14.
// (With the query rows as the tile's rows 128 rows of 9 tokens under 40 take 37.2 with 9 and 38.1 with 6; but ranges of fewer blocks are shorter sums.)
constexpr int kUdRowEndCost = 12, kUdQueryRowsEndCost = 6;

// kN: query rows per KV head that a launch has room for, 32 (up to 8 tokens) or 64.
template <int kN>
struct UdLayout {
  static constexpr int kSlots = kN == 32 ? 3 : 2;  // ring of tiles of K and of V, in turn
  static constexpr int kSets = kN == 32 ? 3 : 1;   // output accumulators that take the tiles in turn
  static constexpr int kColS = 0;                  // scores [128 keys][kN]
  static constexpr int kColO = kN;                 // set i, dims 128 h ..: [128 dims][kN of the weights' hi terms | kN of the lo terms]
  static constexpr int kQChunk = kN * 128;         // bytes of a 64-dim chunk of the query rows
  static constexpr int kPPanel = 128 * 128;        // bytes of 64 columns of the weights
  static_assert(kColO + kSets * 4 * kN <= kUdTmemCols, "tensor memory");
};
template <int kN>
struct UdSmem {
  union {
    alignas(1024) char slot[UdLayout<kN>::kSlots][kUdTileBlocks][kUdHalfBlock];  // K: [block][8-key group][64-d chunk][8 keys][128 B]; V: [block][64-d chunk][16 keys][128 B]
    float acc[kN][kD];  // on clusters: the CTA's sums, once its products are complete
  };
  alignas(1024) char q[4][UdLayout<kN>::kQChunk];            // [64-d chunk][query row][128 B]
  alignas(1024) char w[kN / 32][UdLayout<kN>::kPPanel];      // weights [panel][key][128 B]: kN = 32 hi and lo terms, 64 a panel of each
  alignas(8) unsigned long long full[UdLayout<kN>::kSlots], empty[UdLayout<kN>::kSlots], q_full, q_free, s_full, p_full, o_full, o_free;
  alignas(16) float red[4][kN];  // per warp and query row: maxima, later sums
  alignas(16) float m[kN];       // running maxima, in units of log2(e) * scale
  alignas(16) float f[kN];       // what raising them does to sums so far; at a segment's end what its output is scaled by
  int scan[16];
  int start_b, start_j, abort_flag, begun;
  uint32_t tmem_base;

  __device__ __forceinline__ float2* ml() { return reinterpret_cast<float2*>(w); }  // on clusters, with acc: (max, sum) per query row
};

// What a CTA does for one row: blocks j0, j0 + stride, ... (n of them) of row b, which has nb blocks and len keys.
struct UdSeg {
  int b, j0, n, stride, nb, len;
  __device__ __forceinline__ int tiles() const { return (n + kUdTileBlocks - 1) / kUdTileBlocks; }
  __device__ __forceinline__ int tile_blocks(int t) const { return min(n - t * kUdTileBlocks, kUdTileBlocks); }
  __device__ __forceinline__ bool whole() const { return n == nb; }
  __device__ __forceinline__ bool has_row_end() const { return j0 + (n - 1) * stride == nb - 1; }
};
// The CTA's segments: those of its range, or on clusters (kCluster) its share of the cluster's row.
template <bool kCluster>
struct UdWalk {
  int b, j;
  long long g, g1;
  UdSeg one;
  __device__ __forceinline__ bool next(const DecodeParams& p, UdSeg& s) {
    if constexpr (kCluster) {
      s = one;
      one.n = 0;
      return s.n > 0;
    } else {
      Seg r;
      if (!next_seg(p, b, j, g, g1, r)) return false;
      s = UdSeg{r.b, r.j0, r.j1 - r.j0, 1, r.nb, r.len};
      return true;
    }
  }
};

// A place in the ring: K and V of a tile follow one another.
template <int kSlots>
struct UdRing {
  int at = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void step() {
    if (++at == kSlots) { at = 0; phase ^= 1u; }
  }
};

// ---- warp 5: TMA loads.  `ids`: the first 32 block ids, where they are known already (clusters) --------------------
template <int kN, bool kCluster>
__device__ __forceinline__ void ud_producer(const CUtensorMap* k_map, const CUtensorMap* v_map, const DecodeParams& p, UdSmem<kN>& sm, int kvh,
                                            UdWalk<kCluster> walk, int ids, int lane) {
  const int oob = (int)(p.num_blocks * kBlk);  // a box that starts here is filled with zeros
  uint64_t policy;  // every block is read once: do not let it displace what the L2 is good for
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  auto ids_at = [&](const UdSeg& s, int i) {
    return i + lane < s.n ? p.block_tables[decode_table_base(p, s.b) + s.j0 + (i + lane) * s.stride] : 0;
  };
  UdRing<UdLayout<kN>::kSlots> at;
  bool reuse = false;  // the slot has been used before
  UdSeg s, nxt;
  bool have = walk.next(p, s);
  if (!kCluster && have) ids = ids_at(s, 0);
  while (have) {
    bool more = false;
    int next_first = 0;
    for (int i0 = 0; i0 < s.n; i0 += 32) {  // 32 block ids = 4 tiles at a time
      const int ahead = ids_at(s, i0 + 32);
      const int n = min(s.n - i0, 32);
      const bool bad = lane < n && (ids < 0 || ids >= p.num_blocks);
      if (bad) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
      const int token = bad || lane >= n ? oob : ids * kBlk;
      for (int i = 0; i < n; i += kUdTileBlocks) {
        const int cnt = min(n - i, kUdTileBlocks), mine = __shfl_sync(kFullMask, token, (i + lane) & 31);  // a lane per block
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          if (reuse && !um_wait(&sm.empty[at.at], at.phase ^ 1u, &sm.abort_flag, p.status)) return;
          const uint32_t full = smem_u32(&sm.full[at.at]), dst = smem_u32(sm.slot[at.at]) + lane * kUdHalfBlock;
          if (lane == 0) mbar_arrive_expect_tx(full, (uint32_t)cnt * kUdHalfBlock);
          __syncwarp();
          if (lane < cnt) {
            if (kv == 0) tma_load_k_half(dst, k_map, mine / 8, kvh, full, policy);
            else tma_load_v_half(dst, v_map, mine, kvh, full, policy);
          }
          __syncwarp();
          at.step();
          if (at.at == 0) reuse = true;
        }
      }
      ids = ahead;
      if (i0 == 0) {  // the row behind this one, once the first copies are on their way
        more = walk.next(p, nxt);
        if (more) next_first = ids_at(nxt, 0);
      }
    }
    s = nxt;
    ids = next_first;
    have = more;
  }
}

// ---- warp 4: MMA issue --------------------------------------------------------------------------
// S(t), then O += V(t)^T P(t), tile by tile: the memory delivers K and V of a tile in turn, and either product of one takes less time
// than the bytes of the other.
template <int kN, bool kCluster>
__device__ __forceinline__ void ud_mma_warp(UdSmem<kN>& sm, const DecodeParams& p, uint32_t tmem, UdWalk<kCluster> walk) {
  using L = UdLayout<kN>;
  constexpr uint32_t idesc_s = umma_idesc(kN, false), idesc_o = umma_idesc(2 * kN, true) | kUmmaTransposedA;
  const uint64_t k_desc0 = umma_desc(smem_u32(sm.slot[0]), 16, 4 * 8 * 128);  // keys are rows (groups of 8: 4 KiB apart), dims contracted
  const uint64_t v_desc0 = umma_desc(smem_u32(sm.slot[0]), kBlk * 128, 1024);  // dims are rows (64-d chunks 2 KiB apart), keys contracted
  const uint64_t q_desc = umma_desc(smem_u32(sm.q[0]), 16, 1024);             // query rows in groups of 8
  const uint64_t w_desc = umma_desc(smem_u32(sm.w[0]), L::kPPanel, 1024);     // panels of 64 columns, keys contracted
  UdRing<L::kSlots> at;
  UdSeg s;
  uint32_t tile = 0;
  for (uint32_t seg = 0; walk.next(p, s); ++seg) {
    const int nt = s.tiles();
    for (int t = 0; t < nt; ++t, ++tile) {
      // (rows of keys that the tile does not have are computed from whatever lies there, and masked)
      if (t == 0 && !um_wait(&sm.q_full, seg & 1u, &sm.abort_flag, p.status)) return;
      if (!um_wait(&sm.full[at.at], at.phase, &sm.abort_flag, p.status)) return;
      tc_fence_after_sync();
      if (um_elect_one()) {
        const uint64_t k_desc = k_desc0 + (uint64_t)((at.at * kUdSlotBytes) >> 4);
#pragma unroll
        for (int ks = 0; ks < 16; ++ks)  // 16 dims per MMA: chunk ks / 4, 32 bytes into its swizzled rows
          umma_bf16_ss(tmem + L::kColS, k_desc + (uint64_t)(((ks >> 2) * (8 * 128) + (ks & 3) * 32) >> 4),
                       q_desc + (uint64_t)(((ks >> 2) * L::kQChunk + (ks & 3) * 32) >> 4), idesc_s, ks > 0 ? 1u : 0u);
        umma_commit(smem_u32(&sm.s_full));
        umma_commit(smem_u32(&sm.empty[at.at]));
        if (t == nt - 1) umma_commit(smem_u32(&sm.q_free));
      }
      __syncwarp();
      at.step();
      if (!um_wait(&sm.full[at.at], at.phase, &sm.abort_flag, p.status)) return;
      if (!um_wait(&sm.p_full, tile & 1u, &sm.abort_flag, p.status)) return;
      // the first weighted sum of a segment overwrites O: the segment before must have been read out
      if (t == 0 && seg > 0 && !um_wait(&sm.o_free, (seg - 1) & 1u, &sm.abort_flag, p.status)) return;
      tc_fence_after_sync();
      if (um_elect_one()) {
        const int cnt = s.tile_blocks(t);
        const uint32_t o = tmem + L::kColO + (t % L::kSets) * (4 * kN);
        const uint64_t v_desc = v_desc0 + (uint64_t)((at.at * kUdSlotBytes) >> 4);
        for (int i = 0; i < cnt; ++i) {  // 16 keys per MMA, 128 dims each
          const uint32_t more = (t >= L::kSets || i > 0) ? 1u : 0u;
          const uint64_t wd = w_desc + (uint64_t)((i * 16 * 128) >> 4), vd = v_desc + (uint64_t)((i * kUdHalfBlock) >> 4);
          umma_bf16_ss(o, vd, wd, idesc_o, more);
          umma_bf16_ss(o + 2 * kN, vd + (uint64_t)((kUdHalfBlock / 2) >> 4), wd, idesc_o, more);
        }
        umma_commit(smem_u32(&sm.empty[at.at]));
        if (t == nt - 1) umma_commit(smem_u32(&sm.o_full));
      }
      __syncwarp();
      at.step();
    }
  }
}

// Reduces column c of v over the warp's lanes into lane c's result.
template <class Op>
__device__ __forceinline__ float ud_reduce_columns(float (&v)[32], int lane, Op op) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float keep = up ? v[i + o] : v[i], give = up ? v[i] : v[i + o];
      v[i] = op(keep, __shfl_xor_sync(kFullMask, give, o));
    }
  }
  return v[0];
}
// The four softmax warps meet; whether `mine` holds in any of their threads.
__device__ __forceinline__ bool ud_meet_any(bool mine) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any) : "r"((uint32_t)mine) : "memory");
  return any != 0;
}
__device__ __forceinline__ void ud_sts16(uint32_t at, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// ---- warps 0 - 3: softmax and output.  Thread = key of the tile, then dim of the output ------------------------------
// (A wait that runs out does so for one warp and perhaps not for the next: they leave together, behind a meeting.)
template <int kN, bool kCluster>
__device__ __forceinline__ void ud_softmax_warps(UdSmem<kN>& sm, const DecodeParams& p, uint32_t tmem, int kvh, UdWalk<kCluster> walk, int range,
                                                 int warp, int lane) {
  using L = UdLayout<kN>;
  const int key = warp * 32 + lane, cols = 4 * p.width;
  const float scale_log2 = p.scale * kLog2e;
  const uint32_t w_row = smem_u32(sm.w[0]) + key * 128;
  tmem += (uint32_t)(warp * 32) << 16;
  UdRing<L::kSlots> at;
  UdSeg s;
  uint32_t tile = 0;
  for (uint32_t seg = 0; walk.next(p, s); ++seg) {
    int last[kN / 4];  // per token: its last visible key
#pragma unroll
    for (int k = 0; k < kN / 4; ++k) {
      const int pos = k < p.width ? (p.positions ? p.positions[(long long)s.b * p.width + k] : 0x7fffffff) : -1;
      last[k] = pos < s.len - 1 ? pos : s.len - 1;
    }
    float l[kN];
#pragma unroll
    for (int c = 0; c < kN; ++c) l[c] = 0.f;
    const int nt = s.tiles();
    for (int t = 0; t < nt; ++t, ++tile) {
      at.step();  // V's slot
      const int cnt = s.tile_blocks(t);
      // this thread's key; one of a block that the tile does not have is behind everybody's last one
      const int at_key = (key >> 4) < cnt ? (s.j0 + (t * kUdTileBlocks + (key >> 4)) * s.stride) * kBlk + (key & 15) : 0x7fffffff;
      const bool ok = um_wait(&sm.s_full, tile & 1u, &sm.abort_flag, p.status);
      tc_fence_after_sync();
      float sc[kN];
      bool above = false;
#pragma unroll
      for (int c0 = 0; c0 < kN; c0 += 32) {
        float a[32];
        tmem_ld32(tmem + L::kColS + c0, a);
#pragma unroll
        for (int i = 0; i < 32; ++i) sc[c0 + i] = at_key <= last[(c0 + i) >> 2] ? a[i] : -INFINITY;
      }
      if (t > 0) {
#pragma unroll
        for (int c = 0; c < kN; c += 4) {
          const float4 m4 = *reinterpret_cast<const float4*>(&sm.m[c]);
          above |= sc[c] * scale_log2 > m4.x + kUdRescaleGap || sc[c + 1] * scale_log2 > m4.y + kUdRescaleGap ||
                   sc[c + 2] * scale_log2 > m4.z + kUdRescaleGap || sc[c + 3] * scale_log2 > m4.w + kUdRescaleGap;
        }
      }
      if (ud_meet_any(!ok || t == 0 || above)) {
        // the first tile, or rarely a later one: the tile's maxima; what has been summed so far is brought to the new ones
#pragma unroll
        for (int c0 = 0; c0 < kN; c0 += 32) {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = sc[c0 + i];
          sm.red[warp][c0 + lane] = ud_reduce_columns(v, lane, [](float x, float y) { return fmaxf(x, y); });
        }
        if (ud_meet_any(!ok)) return;
        if (key < kN) {
          const float mx = fmaxf(fmaxf(sm.red[0][key], sm.red[1][key]), fmaxf(sm.red[2][key], sm.red[3][key])) * scale_log2;  // scale > 0
          const float old = t == 0 ? -INFINITY : sm.m[key], m_new = fmaxf(old, mx);
          sm.f[key] = m_new == -INFINITY ? 1.f : ex2_approx(old - m_new);
          sm.m[key] = m_new;
        }
        ud_meet_any(false);
        if (t > 0) {  // (the weighted sums so far are complete: S(t) was issued behind them)
#pragma unroll
          for (int c = 0; c < kN; ++c) l[c] *= sm.f[c];
          const int groups = (t < L::kSets ? t : L::kSets) * 4 * kN / 32;
#pragma unroll 1
          for (int cc = 0; cc < groups; ++cc) {
            float o[32];
            tmem_ld32(tmem + L::kColO + cc * 32, o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] *= sm.f[(cc * 32 + i) & (kN - 1)];
            tmem_st32(tmem + L::kColO + cc * 32, o);
          }
        }
      }
#pragma unroll
      for (int c0 = 0; c0 < kN; c0 += 8) {  // two tokens: 16 bytes of the key's row of hi terms, 16 of lo terms
        if (c0 < cols) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 m2 = *reinterpret_cast<const float2*>(&sm.m[c0 + 2 * e]);
            const float p0 = ex2_approx(fmaf(sc[c0 + 2 * e], scale_log2, m2.x == -INFINITY ? 0.f : -m2.x));
            const float p1 = ex2_approx(fmaf(sc[c0 + 2 * e + 1], scale_log2, m2.y == -INFINITY ? 0.f : -m2.y));
            l[c0 + 2 * e] += p0;
            l[c0 + 2 * e + 1] += p1;
            const __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
            const __nv_bfloat162 r2 = __floats2bfloat162_rn(p0 - __low2float(h), p1 - __high2float(h));
            hi[e] = *reinterpret_cast<const uint32_t*>(&h);
            lo[e] = *reinterpret_cast<const uint32_t*>(&r2);
          }
          const int piece = c0 / 8;
          const uint32_t hi_at = w_row + ((piece ^ (key & 7)) << 4);
          ud_sts16(hi_at, hi[0], hi[1], hi[2], hi[3]);
          ud_sts16(kN == 32 ? w_row + (((piece + 4) ^ (key & 7)) << 4) : hi_at + L::kPPanel, lo[0], lo[1], lo[2], lo[3]);
        }
      }
      if (t == nt - 1 && s.has_row_end() && (s.len & (kBlk - 1))) {
        // V rows of the last block behind the last key weigh nothing, but may hold anything: 0 x infinity is not 0
        if (ud_meet_any(!um_wait(&sm.full[at.at], at.phase, &sm.abort_flag, p.status))) return;
        if (at_key != 0x7fffffff && at_key >= s.len) {
          const uint32_t row = smem_u32(sm.slot[at.at][key >> 4]) + (key & 15) * 128;
          for (int i = 0; i < 32; ++i) ud_sts16(row + (i >> 3) * (kBlk * 128) + (i & 7) * 16, 0u, 0u, 0u, 0u);
        }
      }
      fence_proxy_async_smem();
      tc_fence_before_sync();
      mbar_arrive(smem_u32(&sm.p_full));
      at.step();
    }
    // ---- end of the segment: sums over the keys, then the output or the partial
#pragma unroll
    for (int c0 = 0; c0 < kN; c0 += 32) {
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = l[c0 + i];
      sm.red[warp][c0 + lane] = ud_reduce_columns(v, lane, [](float x, float y) { return x + y; });
    }
    if (ud_meet_any(!um_wait(&sm.o_full, seg & 1u, &sm.abort_flag, p.status))) return;
    const bool final_row = !kCluster && s.whole();
    const int slot_rows = p.width * kHq;
    const long long out_row = final_row ? (long long)s.b * slot_rows : (long long)partial_slot(range, s.j0 == 0) * slot_rows;
    if (key < kN) {
      const float sum = (sm.red[0][key] + sm.red[1][key]) + (sm.red[2][key] + sm.red[3][key]);
      const float2 e = make_float2(sm.m[key] == -INFINITY ? kNegBig : sm.m[key], sum);
      sm.f[key] = final_row ? (sum > 0.f ? 1.f / sum : 0.f) : 1.f;
      if (kCluster) sm.ml()[key] = e;
      else if (!final_row && key < cols) *reinterpret_cast<float2*>(p.part_ml + (out_row + (key >> 2) * kHq + kvh * kG + (key & 3)) * 2) = e;
    }
    ud_meet_any(false);
    tc_fence_after_sync();
    const int sets = nt < L::kSets ? nt : L::kSets;
    float* dst = (final_row ? p.out : p.part_acc) + (out_row + kvh * kG) * kD + key;
#pragma unroll 1
    for (int hc = 0; hc < kN / 4; ++hc) {  // 8 columns of dims 128 h ..
      const int h = hc & 1, c0 = (hc >> 1) * 8;
      if (c0 >= cols) break;
      const uint32_t from = tmem + L::kColO + h * (2 * kN) + c0;
      float o[L::kSets][2][8];
#pragma unroll
      for (int k = 0; k < L::kSets; ++k)
        if (k < sets) {
          tmem_ld8(from + k * (4 * kN), o[k][0]);
          tmem_ld8(from + k * (4 * kN) + kN, o[k][1]);
        }
      tmem_ld_wait();
#pragma unroll
      for (int k = 0; k < L::kSets; ++k)
        if (k < sets) {
          tmem_loaded(o[k][0]);
          tmem_loaded(o[k][1]);
        }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float y = o[0][0][i] + o[0][1][i];
#pragma unroll
        for (int k = 1; k < L::kSets; ++k)
          if (k < sets) y += o[k][0][i] + o[k][1][i];
        if (c0 + i < cols) {
          if (kCluster) sm.acc[c0 + i][h * 128 + key] = y;
          else dst[(((c0 + i) >> 2) * kHq + (i & 3)) * kD + h * 128] = y * sm.f[c0 + i];
        }
      }
    }
    tc_fence_before_sync();  // the next segment's first weighted sums overwrite what was just read
    mbar_arrive(smem_u32(&sm.o_free));
  }
}

// ---- warps 6 and 7: a segment's query rows, as soon as the scores of the segment before have been computed --------
template <int kN, bool kCluster>
__device__ __forceinline__ void ud_query_warps(UdSmem<kN>& sm, const DecodeParams& p, int kvh, UdWalk<kCluster> walk, int tid) {
  const int half = tid >> 5, piece = tid & 31;  // a warp takes every other row, a lane a 16-byte piece of it
  const uint32_t dst = smem_u32(sm.q[piece >> 3]);
  UdSeg s;
  for (uint32_t seg = 0; walk.next(p, s); ++seg) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.q) + ((long long)s.b * p.width * kHq + kvh * kG) * kD) + piece;
#pragma unroll 1
    for (int r0 = 0; r0 < 4 * p.width; r0 += 32) {  // 16 rows in flight (of unused ones the last token's again: nobody reads their scores)
      uint4 u[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int row = r0 + 2 * i + half, tok = min(row >> 2, p.width - 1);
        u[i] = ld_stream_u4(src + (tok * kHq + (row & 3)) * (kD / 8));
      }
      if (r0 == 0 && seg > 0 && !um_wait(&sm.q_free, (seg - 1) & 1u, &sm.abort_flag, p.status)) return;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const int row = r0 + 2 * i + half;
        ud_sts16(dst + row * 128 + (((piece & 7) ^ (row & 7)) << 4), u[i].x, u[i].y, u[i].z, u[i].w);
      }
    }
    fence_proxy_async_smem();
    mbar_arrive(smem_u32(&sm.q_full));
  }
}

// The sums of a cluster's CTAs [query row][dim] and their (max, sum) into the output: rank r takes its share of the float4 pieces.
// Returns what cl_sync_read() asks for.
template <int kN>
__device__ __forceinline__ bool ud_fold_cluster(UdSmem<kN>& sm, const DecodeParams& p, int kvh, int b, int rank, int ctas) {
  const int pieces = 4 * p.width * (kD / 4), per = (pieces + ctas - 1) / ctas;
  float* out = p.out + ((long long)b * p.width * kHq + kvh * kG) * kD;
  bool odd = false;
  for (int i = threadIdx.x; i < per; i += kDecodeThreads) {
    const int piece = rank * per + i, c = piece >> 6, d = (piece & 63) * 4;
    if (piece >= pieces) break;
    float2 e[kUdMaxCluster];
    float4 x[kUdMaxCluster];
    float M = kNegBig, L = 0.f;
#pragma unroll
    for (int r = 0; r < kUdMaxCluster; ++r) {
      e[r] = make_float2(kNegBig, 0.f);
      if (r < ctas) e[r] = cl_ld2(cl_map(sm.ml() + c, r));
      if (!(e[r].y == 0.f)) x[r] = cl_ld4(cl_map(&sm.acc[c][d], r));  // (a CTA that has seen no key left nothing there)
      M = fmaxf(M, e[r].x);
    }
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < kUdMaxCluster; ++r)
      if (!(e[r].y == 0.f)) {
        const float f = ex2_approx(e[r].x - M);
        L = fmaf(e[r].y, f, L);
        y.x = fmaf(x[r].x, f, y.x); y.y = fmaf(x[r].y, f, y.y); y.z = fmaf(x[r].z, f, y.z); y.w = fmaf(x[r].w, f, y.w);
      }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    y = make_float4(y.x * inv, y.y * inv, y.z * inv, y.w * inv);
    odd |= cl_not_finite(y);
    *reinterpret_cast<float4*>(out + ((c >> 2) * kHq + (c & 3)) * kD + d) = y;
  }
  return odd;
}

template <int kN, bool kCluster>
__global__ void __launch_bounds__(kDecodeThreads, 1)
decode_umma_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, DecodeParams p) {
  extern __shared__ unsigned char ud_smem_raw[];
  UdSmem<kN>& sm = *reinterpret_cast<UdSmem<kN>*>((reinterpret_cast<uintptr_t>(ud_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int kvh = kCluster ? blockIdx.y : blockIdx.x & 1, range = blockIdx.x >> 1, ranges = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&k_map)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&v_map)) : "memory");
    sm.start_b = p.batch; sm.start_j = 0; sm.abort_flag = 0; sm.begun = 0;
    for (int i = 0; i < UdLayout<kN>::kSlots; ++i) {
      mbar_init(smem_u32(&sm.full[i]), 1);
      mbar_init(smem_u32(&sm.empty[i]), 1);
    }
    mbar_init(smem_u32(&sm.q_full), 64);
    mbar_init(smem_u32(&sm.q_free), 1);
    mbar_init(smem_u32(&sm.s_full), 1);
    mbar_init(smem_u32(&sm.p_full), 128);
    mbar_init(smem_u32(&sm.o_full), 1);
    mbar_init(smem_u32(&sm.o_free), 128);
    mbar_fence_init();
  }
  // The first blocks of the pair's range, K by the one CTA, V by the other; on clusters likewise the first tile's.
  if constexpr (kCluster) {
    const int j = blockIdx.x + lane * gridDim.x;
    if (warp == 7 && p.early_ctas > 0 && lane < kUdTileBlocks && j < p.table_width) {
      const int len = ld_relaxed_gpu(p.seq_lens + blockIdx.z), id = ld_relaxed_gpu(p.block_tables + (long long)blockIdx.z * p.table_width + j);
      if (len > j * kBlk && id >= 0 && id < p.num_blocks) l2_prefetch((kvh == 0 ? p.k_cache : p.v_cache) + (long long)id * kTileBytes, kTileBytes);
    }
  } else {
    __syncthreads();
    if (warp == 7 && p.early_ctas > 0) prefetch_ahead(p, range, ranges, kUdAheadBlocks, kvh == 0, kvh == 1, &sm.begun, lane);
  }
  pdl_wait();
  if (!kCluster && threadIdx.x == 0) *static_cast<volatile int*>(&sm.begun) = 1;
  UdWalk<kCluster> walk{};
  Partition pt{};
  int ids = 0;
  if constexpr (kCluster) {
    // block ids are requested together with the row's length (the table entry exists whatever the length is)
    const int b = blockIdx.z, ctas = gridDim.x, j0 = blockIdx.x;
    if (warp == 5 && j0 + lane * ctas < p.table_width) ids = p.block_tables[decode_table_base(p, b) + j0 + lane * ctas];
    const int len = decode_row_len(p, b), nb = (len + kBlk - 1) / kBlk;
    walk.one = UdSeg{b, j0, nb > j0 ? (nb - j0 + ctas - 1) / ctas : 0, ctas, nb, len};
    if (threadIdx.x < kN) sm.ml()[threadIdx.x] = make_float2(kNegBig, 0.f);
  } else {
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
    pt = make_partition(total, ranges);
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
    __syncthreads();
    walk.b = sm.start_b; walk.j = sm.start_j; walk.g = g0; walk.g1 = g1;
  }
  if (warp == 4) {  // tensor memory between the wait and the release (umma.cuh)
    tmem_alloc(smem_u32(&sm.tmem_base), kUdTmemCols);
    if (lane == 0) pdl_release();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sm.tmem_base;

  if (warp < 4) ud_softmax_warps<kN>(sm, p, tmem, kvh, walk, range, warp, lane);
  else if (warp == 4) {
    if (!kCluster && kvh == 0 && lane == 0) umma_cuts(p, ranges)[range] = umma_cut(p, pt, range, walk.b, walk.j, walk.g);
    __syncwarp();
    ud_mma_warp<kN>(sm, p, tmem, walk);
  }
  else if (warp == 5) ud_producer<kN>(&k_map, &v_map, p, sm, kvh, walk, ids, lane);
  else ud_query_warps<kN>(sm, p, kvh, walk, threadIdx.x - 192);

  tc_fence_before_sync();
  __syncthreads();
  if (sm.abort_flag) {  // give copies and MMAs in flight time to land before the CTA's memory is released
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    __syncthreads();
  }
  if (warp == 4) tmem_dealloc(tmem, kUdTmemCols);
  if constexpr (kCluster) {
    cl_sync();
    const bool odd = ud_fold_cluster<kN>(sm, p, kvh, blockIdx.z, blockIdx.x, gridDim.x);
    cl_sync_read(odd);  // nobody leaves while its shared memory is being read
  }
}

// One CTA per (boundary between two ranges, query token): the first boundary that cuts a row folds the row from the ranges' partials.
// Runs behind the tile kernel in stream order, so it needs neither counters nor fences, and is told by it what was cut where.  (One
// CTA per row and token, each of which found that out for itself, took 10 - 15 us behind 256 rows and 6 behind 64; one per row that
// folded its tokens in turn 8.2 for 64 rows of 8 tokens: every fold is three round trips to the L2.)  Beside the kernel for 9 - 16
// tokens its CTAs wait in place (with 92 registers, where they do not fit, 5 rows of 9 tokens over 8000 - 12000 keys 35.2 us, so 34.1, 64 of 9
// over 256 - 1024 34.1 and 33.8), which seven parts in flight leave room for; beside the one for fewer tokens, which takes the registers
// and the shared memory of a whole SM, they cannot.
__global__ void __maxnreg__(kUmmaMergeRegs)
decode_umma_merge_kernel(DecodeParams p, int ranges) {
  __shared__ float red[384];
  const int tok = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_wait();
  pdl_release();
  const UmmaCut cut = umma_cuts(p, ranges)[blockIdx.x + 1];
  const int b = cut.b, c_lo = cut.first, c_hi = cut.last;
  if (b < 0) return;
  const int slot_rows = p.width * kHq;
  const long long qbase = (long long)b * p.width;
  int first = c_lo, n = c_hi - c_lo + 1;
  if (n <= 32) {
    fold_parts<true, 7>(p, red, tid, 0, first, c_lo, n, (qbase + tok) * kHq, slot_rows, tok * kHq);
    return;
  }
  // more than 32 parts (a few very long rows): a plain running fold, thread = (head, 8 dims), four parts in flight
  const int h = warp, d0 = lane * 8;
  {
    float M = kNegBig, L = 0.f, acc[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] = 0.f;
    for (int i0 = 0; i0 < n; i0 += 4) {
      float2 e[4];
      float4 x[4][2];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = i0 + k < n;
        const int c = c_lo + (ok ? i0 + k : 0);
        const long long row = ((long long)(2 * c + (c == c_lo ? 1 : 0)) * slot_rows + tok * kHq + h);
        e[k] = ok ? __ldcg(reinterpret_cast<const float2*>(p.part_ml + row * 2)) : make_float2(kNegBig, 0.f);
        const float4* src = reinterpret_cast<const float4*>(p.part_acc + row * kD + d0);
        x[k][0] = ok ? __ldcg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[k][1] = ok ? __ldcg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float Mn = fmaxf(M, e[k].x);
        const float fo = ex2_approx(M - Mn), fn = ex2_approx(e[k].x - Mn);
        M = Mn;
        L = L * fo + e[k].y * fn;
        acc[0] = acc[0] * fo + x[k][0].x * fn; acc[1] = acc[1] * fo + x[k][0].y * fn;
        acc[2] = acc[2] * fo + x[k][0].z * fn; acc[3] = acc[3] * fo + x[k][0].w * fn;
        acc[4] = acc[4] * fo + x[k][1].x * fn; acc[5] = acc[5] * fo + x[k][1].y * fn;
        acc[6] = acc[6] * fo + x[k][1].z * fn; acc[7] = acc[7] * fo + x[k][1].w * fn;
      }
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    float4* o = reinterpret_cast<float4*>(p.out + ((qbase + tok) * kHq + h) * kD + d0);
    o[0] = make_float4(acc[0] * inv, acc[1] * inv, acc[2] * inv, acc[3] * inv);
    o[1] = make_float4(acc[4] * inv, acc[5] * inv, acc[6] * inv, acc[7] * inv);
  }
}

typedef CUresult (*UdEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static UdEncodeTiledFn ud_encode_fn() {
  static UdEncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult res;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &res) != cudaSuccess ||
        res != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return reinterpret_cast<UdEncodeTiledFn>(ptr);
  }();
  return fn;
}

// A cache layer [token, kv head, 256] bf16 seen as {64 dims, token, 64-dim chunk, kv head}: one box of {64, 16, 4, 1}
// is one KV head's half of a block and lands as [chunk][16 tokens][128 B] with the 128-byte swizzle in every panel.
static bool ud_make_v_map(CUtensorMap* map, const void* base, uint64_t tokens) {
  const cuuint64_t dims[4] = {64, tokens, 4, (cuuint64_t)kHkv};
  const cuuint64_t strides[3] = {(cuuint64_t)kTokenBytes, 128, (cuuint64_t)kRowBytes};
  const cuuint32_t box[4] = {64, (cuuint32_t)kBlk, 4, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return ud_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
template <int kChunks>
static bool ud_make_grouped_map(CUtensorMap* map, const void* base, uint64_t tokens) {
  const cuuint64_t dims[5] = {64, 8, 4, tokens / 8, (cuuint64_t)kHkv};
  const cuuint64_t strides[4] = {(cuuint64_t)kTokenBytes, 128, 8 * (cuuint64_t)kTokenBytes, (cuuint64_t)kRowBytes};
  const cuuint32_t box[5] = {64, 8, kChunks, kBlk / 8, 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return ud_encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool grouped_map_cached(CUtensorMap* map, const void* cache_layer, uint64_t tokens, int chunks) {
  return ud_encode_fn() && (chunks == 4 ? tensor_map_cached(map, 4, cache_layer, tokens, ud_make_grouped_map<4>)
                                        : tensor_map_cached(map, 2, cache_layer, tokens, ud_make_grouped_map<2>));
}
bool half_block_maps(CUtensorMap* k_map, CUtensorMap* v_map, const void* k_layer, const void* v_layer, uint64_t tokens) {
  return grouped_map_cached(k_map, k_layer, tokens, 4) && tensor_map_cached(v_map, 3, v_layer, tokens, ud_make_v_map);
}
bool tensor_maps_available() { return ud_encode_fn() != nullptr; }

int launch_decode_umma_query_rows(const DecodeParams& p, int ranges, const CUtensorMap& k_map, const CUtensorMap& v_map, cudaStream_t stream);

template <int kN>
static constexpr int ud_smem_bytes() {
  constexpr int bytes = (int)sizeof(UdSmem<kN>) + 1024;
  static_assert(bytes <= 232448, "the ring exceeds the shared memory of one CTA");
  return bytes;
}
// Clusters of `ctas` CTAs (one to an SM) that fit the current device at once; 0 where the driver does not say.
template <int kN>
static int clusters_that_fit(int ctas) {
  static std::atomic<int> known[kMaxDevices][kUdMaxCluster + 1];  // plus one
  const int dev = current_device();
  if (dev < 0) return 0;
  const int seen = known[dev][ctas].load(std::memory_order_relaxed);
  if (seen > 0) return seen - 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, kHkv, 128);
  cfg.blockDim = dim3(kDecodeThreads, 1, 1);
  cfg.dynamicSmemBytes = ud_smem_bytes<kN>();
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaFuncSetAttribute(decode_umma_kernel<kN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes) != cudaSuccess ||
      cudaFuncSetAttribute(decode_umma_kernel<kN, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, decode_umma_kernel<kN, true>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  known[dev][ctas].store(n + 1, std::memory_order_relaxed);
  return n;
}

// CTAs per cluster for this call, or 0 for ranges.  One cluster per row and KV head, as many CTAs each as find a place together, four
// blocks of the table's width or more to each.  Measured at 1 - 200 rows, 5, 8 and 9 tokens, rows of 1/4 - 1 and of 1/32 - 1/8 of the
// table (us, attention alone, ranges : clusters): up to 48 blocks per CTA the clusters are ahead, 2 rows under 256 blocks 17.5 : 11.7 and
// 12.0 : 8.4, 16 under 128 22.1 : 17.3 and 13.3 : 9.0, 64 under 32 23.1 : 18.0 and 17.3 : 9.7, 70 under 50 27.3 : 26.3 and 17.0 : 12.0; beyond
// the ranges' equal shares win on full tables, 47 under 50 23.3 : 24.5, 47 under 60 24.5 : 26.8, 24 under 128 (64 per CTA) 24.7 : 25.2.  Where
// the clusters do not fit at once the second wave costs more than the ranges do (100 rows under 40 30.0 : 36.4, 256 under 16 38.0 : 51.1).
// More than 8 tokens: two CTAs at least, 8 rows under 64 blocks 17.1 : 13.9 and 12.4 : 10.3, 36 under 40 23.8 : 19.8 and 14.6 : 12.0; with one, 41 rows
// under 22 20.0 : 21.0 and 11.3 : 14.2, 64 under 64 32.1 : 35.0.
static int umma_cluster(const DecodeParams& p, int sms) {
  const int groups = kHkv * p.batch;
  const bool wide = p.width > 8;
  if (p.batch > sms / kHkv || p.table_width < 1) return 0;
  int c = (p.table_width + 3) / 4;
  c = c < kUdMaxCluster ? c : kUdMaxCluster;
  while (c > 1 && (c * groups > sms || (wide ? clusters_that_fit<64>(c) : clusters_that_fit<32>(c)) < groups)) --c;
  return (p.table_width + c - 1) / c <= (wide ? 40 : 48) && (c > 1 || !wide) ? c : 0;
}

template <int kN>
static int launch_on_clusters(const CUtensorMap& k_map, const CUtensorMap& v_map, const DecodeParams& p, int ctas, cudaStream_t stream) {
  static PerDeviceFlags opted_in;
  return launch_clusters(decode_umma_kernel<kN, true>, opted_in, p, dim3(ctas), kHkv, kDecodeThreads, ud_smem_bytes<kN>(), stream, k_map, v_map, p);
}
static int launch_on_ranges(const CUtensorMap& k_map, const CUtensorMap& v_map, const DecodeParams& p, int ranges, cudaStream_t stream) {
  static PerDeviceFlags opted_in;
  if (!once_per_device(opted_in, [](int) {
        return cudaFuncSetAttribute(decode_umma_kernel<32, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, ud_smem_bytes<32>()) == cudaSuccess;
      }))
    return NVJ_ERR_LAUNCH;
  launch_after(decode_umma_kernel<32, false>, 2 * ranges, kDecodeThreads, ud_smem_bytes<32>(), stream, k_map, v_map, p);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

// p as launch_decode_wide takes it (width 2..16, carved workspace whose partial area holds ws_slots(decode_wide_num_ctas())
// slots of width * kHq rows).  NVJ_ERR_UNSUPPORTED: no tensor-map encoder, a scale that is not positive (row maxima are
// taken before scaling), the packed or the appending form.
int launch_decode_umma(const DecodeParams& p, cudaStream_t stream) {
  if (p.width < 1 || p.width > kUdMaxWidth || p.num_blocks < 1 || (p.num_blocks + 1) * kBlk > 0x7fffffffLL || !ud_encode_fn() ||
      !(p.scale > 0.f) || p.packed_rows || p.new_k || p.kv_indptr)
    return NVJ_ERR_UNSUPPORTED;
  const int ctas = decode_wide_num_ctas();
  if (ctas < 2) return NVJ_ERR_LAUNCH;
  const int ranges = ctas / 2;
  CUtensorMap k_map, v_map;
  if (!half_block_maps(&k_map, &v_map, p.k_cache, p.v_cache, (uint64_t)p.num_blocks * kBlk)) return NVJ_ERR_UNSUPPORTED;
  DecodeParams q = p;
  q.row_end_cost = p.width > 8 ? kUdQueryRowsEndCost : kUdRowEndCost;
  q.early_ctas = ahead_ctas(p, ctas);
  const int cluster = umma_cluster(p, ctas);
  int rc;
  if (cluster > 0) rc = p.width > 8 ? launch_on_clusters<64>(k_map, v_map, q, cluster, stream) : launch_on_clusters<32>(k_map, v_map, q, cluster, stream);
  else rc = p.width > 8 ? launch_decode_umma_query_rows(q, ranges, k_map, v_map, stream) : launch_on_ranges(k_map, v_map, q, ranges, stream);
  if (rc != NVJ_OK || cluster > 0) return rc;
  if (ranges < 2) return NVJ_OK;
  launch_after(decode_umma_merge_kernel, dim3(ranges - 1, p.width), kDecodeThreads, 0, stream, q, ranges);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

}  // namespace nvj
