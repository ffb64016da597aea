// Paged GQA decode attention, one query token per row, for batches whose K and V stream from HBM for a long time: the decode
// step proper with the optional fused append, and the decode rows of a packed batch.  bf16, 16-token blocks, 2 KV heads x 4
// query heads, head_dim 256.
//
// What bounds it: HBM, and on long launches the 1000 W that the board may draw (a plain sum over memory takes 772 W at 6.5 TB/s,
// so the arithmetic has ~230 W to itself).  The work around the bytes is therefore kept small, not only hidden:
//   * Every K/V byte crosses HBM once: one TMA box of 16 KiB per block of K and of V (both KV heads), evict-first, into a ring
//     of 3 boxes for each of four walkers (192 KiB), [kv head][64-dim chunk][16 tokens][128 B] with the 128-byte swizzle.
//   * Eight consumer warps: warp = (walker, kv head).  A walker takes every fourth block of the CTA's range; each byte of a box is
//     read from shared memory once.  Both products are transposed (S^T = K Q^T, O^T = V^T P^T), so that the four heads of the
//     group are half of the N = 8 columns and the weights as hi + lo fill them: 32 mma.sync and 32 ldmatrix per block and head.
//     (The untransposed form that rows of several tokens use spends 128 and 48 on it: four of its sixteen tile rows are real, and
//     two warps repeat each block's scores.)
//   * A ninth warp feeds the ring: it walks the rows, holds the block ids of the next 32 blocks (and asks for the 32 behind them
//     and for the next row's in advance) and waits for a slot to be given back.  Nobody else waits for anything but its own
//     copies, except at the end of a row, where the walkers' sums meet in shared memory.
// The split over CTAs, the partials and their fold are the CUDA-core kernel's (decode_parts.cuh).
// Measured (us per launch, back to back; before: the untransposed form): 128 rows of 8192 - 32768 keys 906 -> 775 once the board
// has warmed up (the form before ran at its power limit), 200 of 3000 - 9000 368 -> 368, 128 of 512 - 4096 101 -> 96, 256 of 128 - 1024
// 65 -> 55, 8 of 8192 - 32768 63.4 -> 61.5, one of 32768 26.1 -> 25.2; what the
// prefetch ahead of the wait gives stands at kStAheadBlocks.
// Semantics: nanovllm_jax/kv_cache.py:852-998 for width-1 queries; the fused append follows
// nanovllm_jax/kernels/full_attention_triton.py:373-485.

#include <cuda.h>

#include "decode_cluster.cuh"
#include "umma.cuh"

namespace nvj {

// Development aid, compiled in only with -DNVJ_PHASE_TIMING: every CTA stamps the global timer at the kernel's phase boundaries,
// and nvj_debug_phase_ns copies the stamps out.
#ifdef NVJ_PHASE_TIMING
__device__ unsigned long long g_phase_ns[256][9];  // slots 0-6: stamps; 7: the SM the CTA ran on; 8: its number of blocks
#define NVJ_PHASE_NOTE(thread, i, v) do { if (threadIdx.x == (thread)) g_phase_ns[blockIdx.x][i] = (v); } while (0)
#else
#define NVJ_PHASE_NOTE(thread, i, v) do { } while (0)
#endif
#define NVJ_PHASE(i) NVJ_PHASE_NOTE(0, i, global_timer_ns())

constexpr int kStWalkers = 4;
constexpr int kStSlots = 3;  // boxes per walker: K and V of a block alternate
// Two warpgroups of consumers and one that holds the producer's warp.  A thread gets 168 registers at launch; the consumers, which
// want more (any spill costs a launch 1 - 3 us), take what the third group gives up: 256 x 240 + 128 x 24 = 384 x 168.
constexpr int kStThreads = kDecodeThreads + 128;
constexpr int kStConsumerRegs = 240, kStProducerRegs = 24;
static_assert(kDecodeThreads * kStConsumerRegs + 128 * kStProducerRegs <= kStThreads * 168, "more registers than the launch has");
constexpr int kStPitch = kD + 4;  // floats between the heads of a warp's sums: conflict-free stores
constexpr int kStRowEndCost = 9;  // blocks that a row end costs a CTA (decode_parts.cuh): 32 rows of 512 - 4096 keys 34.1 us with 1, 33.3 with 6, 32.5 with 9

// Blocks of a CTA's range that are prefetched ahead of the wait (prefetch_ahead).  Passes back to back, each behind another of this kernel,
// without it : with it: 8 rows of 8192 - 32768 keys 60.1 : 55.9 us, 24 of 4096 - 16384 83.7 : 79.1, 32 of 2000 - 8000 58.4 : 53.0, one row of 20000
// and 128 of 8192 - 32768 the same (16.9 : 16.8, 783 : 785); behind a kernel that ends all at once there is nothing to gain (63.9 : 63.6).
// With six blocks the first case is 0.7 us later, with 18 as well, with 26 1.6.
constexpr int kStAheadBlocks = 12;

struct StreamSmem {
  alignas(1024) char tiles[kStWalkers][kStSlots][kTileBytes];
  union {
    alignas(16) float xo[kHkv][kStWalkers][kG][kStPitch];  // the warps' sums at the end of a row
    float red[384];                                        // scratch of fold_parts, once those have been read
  };
  float2 ml[kHkv][kStWalkers][kG];
  alignas(8) unsigned long long full_bar[kStWalkers][kStSlots], empty_bar[kStWalkers][kStSlots];
  int in_pool[kStWalkers][kStSlots];  // whether the slot's block lies in the pool (read with K)
  int scan[16];
  int start_b, start_j, is_last, abort_flag, begun;
};

// A position in one walker's ring.
struct StCursor {
  int slot = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ void step() {
    if (++slot == kStSlots) { slot = 0; phase ^= 1u; }
  }
};

template <bool kWindow>
__device__ __forceinline__ void st_producer(const CUtensorMap* k_map, const CUtensorMap* v_map, const DecodeParams& p, StreamSmem& sm,
                                            int b, int j, long long g, long long g1, int lane) {
  uint64_t policy;  // every block is read once: do not let it displace what the L2 is good for
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  auto ids_at = [&](const Seg& s, int jb) { return jb + lane < s.j1 ? p.block_tables[decode_table_base(p, s.b) + jb + lane] : -1; };
  StCursor at;  // of the walkers that are being served: all four have taken part equally often when `wk` wraps
  int wk = 0;
  bool reuse = false;  // the slot has been used before
  Seg s, nxt;
  bool have = next_seg<kWindow>(p, b, j, g, g1, s);
  int ids = have ? ids_at(s, s.j0) : -1;
  while (have) {
    bool more = false;
    int next_first = -1;
    for (int jb = s.j0; jb < s.j1; jb += 32) {
      const int ahead = ids_at(s, jb + 32);
      const int n = s.j1 - jb < 32 ? s.j1 - jb : 32;
      if (lane < n && (ids < 0 || ids >= p.num_blocks)) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
      for (int i = 0; i < n; ++i) {
        const int blk = __shfl_sync(kFullMask, ids, i);
        const bool ok = blk >= 0 && blk < p.num_blocks;
        StCursor c = at;
        bool again = reuse;
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          // (phase c.phase of the slot's full barrier follows the release of phase c.phase ^ 1)
          if (again && !mbar_wait(smem_u32(&sm.empty_bar[wk][c.slot]), c.phase ^ 1u, &sm.abort_flag, p.status)) return;
          if (lane == 0) {
            const uint32_t full = smem_u32(&sm.full_bar[wk][c.slot]);
            if (ok) {
              if (kv == 0) sm.in_pool[wk][c.slot] = 1;
              mbar_arrive_expect_tx(full, kTileBytes);
              tma_load_block(smem_u32(sm.tiles[wk][c.slot]), kv ? v_map : k_map, blk * kBlk, full, policy);
            } else {
              if (kv == 0) sm.in_pool[wk][c.slot] = 0;
              mbar_arrive(full);
            }
          }
          if (!reuse && wk == 0 && kv == 0) NVJ_PHASE_NOTE(kDecodeThreads, 3, global_timer_ns());
          __syncwarp();
          c.step();
          if (c.slot == 0) again = true;
        }
        if (++wk == kStWalkers) { wk = 0; at = c; reuse = again; }
      }
      ids = ahead;
      if (jb == s.j0) {  // the row behind this one, once the first copies are on their way
        more = next_seg<kWindow>(p, b, j, g, g1, nxt);
        if (more) next_first = ids_at(nxt, nxt.j0);
      }
    }
    s = nxt;
    ids = next_first;
    have = more;
  }
}

// One warp's share of a row: sums over the blocks it has seen, columns of the transposed tiles (a lane holds heads (2 t) & 3 and
// (2 t + 1) & 3, dims 16 n + g and 16 n + g + 8; lanes t >= 2 what the weights' rounding left over).
struct StState {
  float o[16][4];
  float m[2], l[2];
};

// The walkers' sums into the output row or the CTA's partial, which is then counted in.
__device__ __forceinline__ void st_finish_segment(const DecodeParams& p, StreamSmem& sm, const Seg& s, StState& st, int warp, int lane,
                                                  const Partition& pt) {
  const int g = lane >> 2, t = lane & 3, kvh = warp & 1, wk = warp >> 1;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    st.l[c] += __shfl_xor_sync(kFullMask, st.l[c], 4);
    st.l[c] += __shfl_xor_sync(kFullMask, st.l[c], 8);
    st.l[c] += __shfl_xor_sync(kFullMask, st.l[c], 16);
    if (lane < 2) sm.ml[kvh][wk][2 * t + c] = make_float2(st.m[c], st.l[c]);
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)  // both terms of a column are added: of two tiles a lane keeps one and gives the other away
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float keep = t < 2 ? st.o[2 * k][e] : st.o[2 * k + 1][e], give = t < 2 ? st.o[2 * k + 1][e] : st.o[2 * k][e];
      sm.xo[kvh][wk][2 * (t & 1) + (e & 1)][(2 * k + (t >> 1)) * 16 + g + 8 * (e >> 1)] = keep + __shfl_xor_sync(kFullMask, give, 2);
    }
  named_bar_sync(1, kDecodeThreads);
  // warp = head: the four walkers' sums, 2 x 4 dims per lane
  const bool whole_row = (s.j0 == 0 && s.j1 == s.nb);
  const long long qi = decode_query_index(p, s.b);
  const int kv = warp >> 2, h = warp & 3;
  float M = kNegBig, L = 0.f;
#pragma unroll
  for (int w = 0; w < kStWalkers; ++w) M = fmaxf(M, sm.ml[kv][w][h].x);
  float4 y[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
#pragma unroll
  for (int w = 0; w < kStWalkers; ++w) {
    const float2 e = sm.ml[kv][w][h];
    const float f = ex2_approx(e.x - M);
    L = fmaf(e.y, f, L);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const float4 x = *reinterpret_cast<const float4*>(&sm.xo[kv][w][h][d * 128 + lane * 4]);
      y[d].x = fmaf(x.x, f, y[d].x); y[d].y = fmaf(x.y, f, y[d].y); y[d].z = fmaf(x.z, f, y[d].z); y[d].w = fmaf(x.w, f, y[d].w);
    }
  }
  const float inv = whole_row ? (L > 0.f ? 1.f / L : 0.f) : 1.f;
  const long long row = whole_row ? qi * kHq + warp : (long long)partial_slot(blockIdx.x, s.j0 == 0) * kHq + warp;
  float* dst = (whole_row ? p.out : p.part_acc) + row * kD + lane * 4;
#pragma unroll
  for (int d = 0; d < 2; ++d)
    *reinterpret_cast<float4*>(dst + d * 128) = make_float4(y[d].x * inv, y[d].y * inv, y[d].z * inv, y[d].w * inv);
  if (whole_row) {
    named_bar_sync(1, kDecodeThreads);  // the exchange buffer is free again
    return;
  }
  if (lane == 0) *reinterpret_cast<float2*>(p.part_ml + row * 2) = make_float2(M, L);
  finish_shared_row<8>(p, sm.red, sm.is_last, s, pt, qi, warp * 32 + lane);
}

template <bool kWindow>
__device__ __forceinline__ void st_consumer(const DecodeParams& p, StreamSmem& sm, const Partition& pt, int b, int j, long long g0,
                                            long long g1, int warp, int lane) {
  const int g = lane >> 2, t = lane & 3, kvh = warp & 1, wk = warp >> 1;
  const float scale_log2 = p.scale * kLog2e;
  // offsets of this lane's ldmatrix rows inside a box; chunks of 64 dims are 2 KiB apart, 16-byte pieces XORed with the token
  const uint32_t k_off = kvh * 8192 + ((lane & 7) + ((lane >> 3) & 1) * 8) * 128, k_piece = ((lane >> 4) ^ (lane & 7)) << 4;
  const uint32_t v_off = kvh * 8192 + ((lane & 7) + (lane >> 4) * 8) * 128, v_piece = (((lane >> 3) & 1) ^ (lane & 7)) << 4;
  long long gg = g0;
  int it = 0;  // real blocks of the range so far: block i belongs to walker i % 4
  StCursor at;
  Seg s;
  while (next_seg<kWindow>(p, b, j, gg, g1, s)) {
    const long long qi = decode_query_index(p, s.b);
    uint32_t qb[16][2];  // Q^T as the B operand: column g = head g & 3
    {
      const char* q = static_cast<const char*>(p.q) + ((qi * kHq + kvh * kG + (g & 3)) * kD) * 2;
#pragma unroll
      for (int ks = 0; ks < 16; ++ks) {
        qb[ks][0] = *reinterpret_cast<const uint32_t*>(q + ks * 32 + t * 4);
        qb[ks][1] = *reinterpret_cast<const uint32_t*>(q + ks * 32 + 16 + t * 4);
      }
    }
    StState st;
#pragma unroll
    for (int n = 0; n < 16; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) st.o[n][e] = 0.f;
    st.m[0] = st.m[1] = kNegBig;
    st.l[0] = st.l[1] = 0.f;
    // Fused append.  The CTA that owns block min(pos / 16, nb - 1) of the row writes the new K/V row (one warp per KV head); its
    // copy of that block may race with the store, so the warps that read the block overwrite the row in the staged box, from the
    // same source, once the copy has landed: no fence is needed and nothing waits for the store.
    int patch_j = -1, patch_t = 0;
    if (p.new_k) {
      const int pos = p.pre_append ? p.seq_lens[s.b] : p.positions[s.b];
      const int jt = pos >> 4;
      const int jw = jt < s.nb - 1 ? jt : s.nb - 1;
      if (pos >= 0 && jw >= s.j0 && jw < s.j1) {
        const long long tgt = jt < p.table_width ? (long long)p.block_tables[decode_table_base(p, s.b) + jt] : -1;
        if (tgt >= 0 && tgt < p.num_blocks) {
          if (wk == 0) {
            const long long src = (long long)s.b * kTokenBytes + kvh * kRowBytes + lane * 16;
            const long long dst = (tgt * kBlk + (pos & 15)) * kTokenBytes + kvh * kRowBytes + lane * 16;
            *reinterpret_cast<uint4*>(const_cast<char*>(p.k_cache) + dst) =
                *reinterpret_cast<const uint4*>(static_cast<const char*>(p.new_k) + src);
            *reinterpret_cast<uint4*>(const_cast<char*>(p.v_cache) + dst) =
                *reinterpret_cast<const uint4*>(static_cast<const char*>(p.new_v) + src);
          }
          if (jt == jw && pos < s.len) { patch_j = jw; patch_t = pos & 15; }
        } else if (warp == 0 && lane == 0) {
          atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
        }
      }
    }
    // lane l carries 16-byte piece l of the KV head's 512-byte row; the source is cache-hot
    auto patch = [&](char* tile, const void* fresh) {
      const uint32_t off = kvh * 8192 + (lane >> 3) * 2048 + patch_t * 128 + (((lane & 7) ^ (patch_t & 7)) << 4);
      *reinterpret_cast<uint4*>(tile + off) =
          *reinterpret_cast<const uint4*>(static_cast<const char*>(fresh) + (long long)s.b * kTokenBytes + kvh * kRowBytes + lane * 16);
      fence_proxy_async_all();  // the slot is refilled by a copy later
      __syncwarp();
    };
    for (int jb = s.j0 + ((wk - it) & (kStWalkers - 1)); jb < s.j1; jb += kStWalkers) {
      mbar_wait(smem_u32(&sm.full_bar[wk][at.slot]), at.phase, &sm.abort_flag, p.status);  // K has landed
      if (it + jb == s.j0) NVJ_PHASE(4);
      const int left = sm.in_pool[wk][at.slot] ? s.len - jb * kBlk : 0;  // keys of the block that are attended; none of a bad id's
      float sc[4];
      {
        if (jb == patch_j) patch(sm.tiles[wk][at.slot], p.new_k);
        const uint32_t base = smem_u32(sm.tiles[wk][at.slot]) + k_off;
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};  // two chains of eight
#pragma unroll
        for (int ks = 0; ks < 16; ks += 2) {
          uint32_t a[4];
          cm_ldsm4(base + (ks >> 2) * 2048 + (k_piece ^ ((ks & 3) << 5)), a);
          cm_mma<__nv_bfloat16>(s0, a, qb[ks][0], qb[ks][1]);
          cm_ldsm4(base + (ks >> 2) * 2048 + (k_piece ^ (((ks + 1) & 3) << 5)), a);
          cm_mma<__nv_bfloat16>(s1, a, qb[ks + 1][0], qb[ks + 1][1]);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&sm.empty_bar[wk][at.slot]));
        at.step();
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[e] = g + (e >> 1) * 8 < left ? (s0[e] + s1[e]) * scale_log2 : kNegBig;
      }
      float alpha[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float mx = fmaxf(sc[c], sc[c + 2]);
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 16));
        const float mn = fmaxf(st.m[c], mx);
        alpha[c] = ex2_approx(st.m[c] - mn);
        st.m[c] = mn;
        st.l[c] *= alpha[c];
      }
      if (__any_sync(kFullMask, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          st.o[n][0] *= alpha[0]; st.o[n][1] *= alpha[1];
          st.o[n][2] *= alpha[0]; st.o[n][3] *= alpha[1];
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[e] = ex2_approx(sc[e] - (st.m[e & 1] <= kNegBig ? 0.f : st.m[e & 1]));  // nothing attended yet: 0
      st.l[0] += sc[0] + sc[2];
      st.l[1] += sc[1] + sc[3];
      const uint32_t b0 = cm_transpose(cm_pack<__nv_bfloat16>(sc[0], sc[1], t >= 2));
      const uint32_t b1 = cm_transpose(cm_pack<__nv_bfloat16>(sc[2], sc[3], t >= 2));
      mbar_wait(smem_u32(&sm.full_bar[wk][at.slot]), at.phase, &sm.abort_flag, p.status);  // V has landed
      if (left > 0) {  // (a block that was not fetched leaves the slot's old contents)
        if (jb == patch_j) patch(sm.tiles[wk][at.slot], p.new_v);
        if (left < kBlk) {  // rows behind the last key weigh nothing, but may hold anything: 0 x infinity is not 0
          for (int r = left; r < kBlk; ++r)
            *reinterpret_cast<uint4*>(sm.tiles[wk][at.slot] + kvh * 8192 + (lane >> 3) * 2048 + r * 128 + (lane & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
          fence_proxy_async_all();
          __syncwarp();
        }
        const uint32_t base = smem_u32(sm.tiles[wk][at.slot]) + v_off;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
          uint32_t a[4];
          cm_ldsm4_t(base + (n >> 2) * 2048 + (v_piece ^ ((n & 3) << 5)), a);
          cm_mma<__nv_bfloat16>(st.o[n], a, b0, b1);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&sm.empty_bar[wk][at.slot]));
      at.step();
    }
    it += s.j1 - s.j0;
    NVJ_PHASE(5);
    st_finish_segment(p, sm, s, st, warp, lane, pt);
    NVJ_PHASE(6);
    NVJ_PHASE_NOTE(0, 8, (unsigned long long)it);
  }
}

// kWindow: decode_row_len.
template <bool kWindow>
__global__ void __launch_bounds__(kStThreads, 1)
decode_stream_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map, DecodeParams p) {
  extern __shared__ unsigned char st_smem_raw[];
  StreamSmem& sm = *reinterpret_cast<StreamSmem*>((reinterpret_cast<uintptr_t>(st_smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int grid = gridDim.x;
  const bool counts = threadIdx.x < kDecodeThreads;  // the producer's warp joins the scans with nothing to add

  NVJ_PHASE(0);
#ifdef NVJ_PHASE_TIMING
  unsigned smid;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
  NVJ_PHASE_NOTE(0, 7, (unsigned long long)smid);
#endif
  // The kernel opens with three dependent trips to memory (lengths -> block ids -> K/V blocks).  While the first is under way, pull
  // what the others will need towards the SM: the tensor maps, and this CTA's share of the block tables into the L2 (all CTAs
  // together cover the tables, so the second trip ends in the L2 for everyone).
  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&k_map)) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&v_map)) : "memory");
    for (int w = 0; w < kStWalkers; ++w)
      for (int i = 0; i < kStSlots; ++i) {
        mbar_init(smem_u32(&sm.full_bar[w][i]), 1);
        mbar_init(smem_u32(&sm.empty_bar[w][i]), kHkv);
      }
    mbar_fence_init();
    sm.start_b = p.batch; sm.start_j = 0; sm.abort_flag = 0; sm.is_last = 0; sm.begun = 0;
  }
  __syncthreads();
  if (warp == kDecodeThreads / 32 + 1 && p.early_ctas > 0) prefetch_ahead(p, blockIdx.x, grid, kStAheadBlocks, true, true, &sm.begun, lane);
  pdl_wait();
  pdl_release();
  if (threadIdx.x == 0) *static_cast<volatile int*>(&sm.begun) = 1;
  if (!p.kv_indptr && counts) {
    const long long lines = ((long long)p.batch * p.table_width * (long long)sizeof(int32_t) + 127) / 128;
    const long long line = (long long)blockIdx.x * kDecodeThreads + threadIdx.x;
    if (line < lines) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p.block_tables) + line * 128));
  }
  // ---- pass 1: total number of blocks; zero the output of inactive rows
  int mine = 0, first_n = 0;
  for (int base = 0; base < p.batch; base += kDecodeThreads) {
    const int b = counts ? base + (int)threadIdx.x : p.batch;
    int len = 0;
    if (b < p.batch) len = decode_row_len<kWindow>(p, b);
    if (base == 0) first_n = blocks_in_sequence(p, (len + kBlk - 1) / kBlk);
    mine += blocks_in_sequence(p, (len + kBlk - 1) / kBlk);
    // rows without keys get zeros; in a packed batch only the rows this pass owns (one query token) are touched
    const bool mine_to_zero = b < p.batch && len <= 0 && (b % grid) == (int)blockIdx.x &&
                              (!p.packed_rows || p.query_start_loc[b + 1] - p.query_start_loc[b] == 1);
    const unsigned idle = __ballot_sync(kFullMask, mine_to_zero);
    for (unsigned m = idle; m; m &= m - 1) {
      const int bb = base + (warp << 5) + (__ffs(m) - 1);
      float4* o = reinterpret_cast<float4*>(p.out + decode_query_index(p, bb) * kHq * kD);
      for (int i = lane; i < kHq * kD / 4; i += 32) o[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  int total = 0;
  const int incl = cta_inclusive_scan(mine, sm.scan, total);
  if (total == 0) return;
  const Partition pt = make_partition(total, grid);
  if ((int)blockIdx.x >= pt.n) return;
  const long long g0 = pt.start(blockIdx.x);
  const long long g1 = pt.start(blockIdx.x + 1);
  if (g0 == g1) return;
  NVJ_PHASE(1);

  // ---- pass 2: locate (row, block) of g0
  long long carry = 0;
  if (p.batch <= kDecodeThreads) {  // one row per thread: the scan of pass 1 has the answer already
    const long long excl = incl - first_n;
    if (counts && first_n > 0 && excl <= g0 && g0 < excl + first_n) { sm.start_b = threadIdx.x; sm.start_j = (int)(g0 - excl); }
    carry = g0 + 1;  // skips the loop below
  }
  for (int base = 0; base < p.batch && carry <= g0; base += kDecodeThreads) {
    const int b = counts ? base + (int)threadIdx.x : p.batch;
    int n = 0;
    if (b < p.batch) n = blocks_in_sequence(p, (decode_row_len<kWindow>(p, b) + kBlk - 1) / kBlk);
    int chunk_total = 0;
    const long long excl = carry + cta_inclusive_scan(n, sm.scan, chunk_total) - n;
    if (n > 0 && excl <= g0 && g0 < excl + n) { sm.start_b = b; sm.start_j = (int)(g0 - excl); }
    carry += chunk_total;
  }
  __syncthreads();
  NVJ_PHASE(2);
  if (warp >= kDecodeThreads / 32) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kStProducerRegs));
    if (warp == kDecodeThreads / 32) st_producer<kWindow>(&k_map, &v_map, p, sm, sm.start_b, sm.start_j, g0, g1, lane);
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kStConsumerRegs));
    st_consumer<kWindow>(p, sm, pt, sm.start_b, sm.start_j, g0, g1, warp, lane);
  }
  __syncthreads();
  // Only after a timeout can copies still be in flight with nobody waiting for them: hold the CTA's shared memory meanwhile.
  if (sm.abort_flag) {
    const unsigned long long t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
}

// One query token per row; p as launch_decode_wide takes it.
int launch_decode_stream(const DecodeParams& p, cudaStream_t stream) {
  int n = decode_wide_num_ctas();
  if (n <= 0) return NVJ_ERR_LAUNCH;
  if (p.cta_limit > 0 && p.cta_limit < n) n = p.cta_limit;
  DecodeParams q = p;
  q.row_end_cost = kStRowEndCost;
  if (!p.new_k && p.positions) {  // keys behind a row's position are not attended
    q.cap_positions = p.positions;
    q.positions = nullptr;
  }
  CUtensorMap k_map, v_map;
  if (!block_map_cached(&k_map, p.k_cache, (uint64_t)p.num_blocks * kBlk) || !block_map_cached(&v_map, p.v_cache, (uint64_t)p.num_blocks * kBlk))
    return NVJ_ERR_UNSUPPORTED;
  static PerDeviceFlags smem_opted_in;
  constexpr int kSmemBytes = (int)sizeof(StreamSmem) + 1024;
  static_assert(kSmemBytes <= 232448, "the ring exceeds the shared memory of one CTA");
  if (!once_per_device(smem_opted_in, [](int) {
        return cudaFuncSetAttribute(decode_stream_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) == cudaSuccess &&
               cudaFuncSetAttribute(decode_stream_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) == cudaSuccess;
      }))
    return NVJ_ERR_LAUNCH;
  q.early_ctas = ahead_ctas(q, n);
  auto* kernel = q.max_len > 0 || q.cap_positions ? decode_stream_kernel<true> : decode_stream_kernel<false>;
  launch_after(kernel, n, kStThreads, kSmemBytes, stream, k_map, v_map, q);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

}  // namespace nvj

#ifdef NVJ_PHASE_TIMING
extern "C" int nvj_debug_phase_ns(unsigned long long* host_out) {  // [256][9]
  return cudaMemcpyFromSymbol(host_out, nvj::g_phase_ns, sizeof(nvj::g_phase_ns)) == cudaSuccess ? 0 : 1;
}
#endif
