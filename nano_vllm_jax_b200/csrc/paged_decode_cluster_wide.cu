// Paged GQA decode attention for rows of 2 - 4 query tokens (speculative verification) on thread-block clusters: few rows, short
// contexts, for which the streaming kernels' fixed costs (~13 us: scan, ring of block ids, fold) are most of the time.
//
// One cluster of C CTAs per row; a CTA takes every C-th block of the row, both KV heads of it, so K/V cross HBM once for all
// of a row's tokens.  As in the width-1 form (paged_decode_cluster.cu) both products are taken transposed, the 4 x width
// query rows of a KV head in the N = 8 columns of ceil(width / 2) tiles:
//   S^T = K Q^T: M = 16 keys, O^T = V^T P^T: M = 16 dims; the weights enter as two bf16 terms (hi + lo).
// Warp (h, dh): KV head h, both computing the block's scores over all dims (a third of the work, repeated by the two), each
// accumulating its half dh of the output dims.  The pair of warps of a head copies that head's K and V rows and shares them;
// the next block's K rows are requested when both have their scores, its V rows after the weighted sums.  Q lies in shared
// memory (its fragments for two tiles do not fit beside the accumulators).
// Bound by latency: a CTA's blocks follow each other, one K and one V block in shared memory.  Measured (us per launch, the
// better streaming form -> this one): 2 tokens, one row of 1024 keys 14.1 -> 8.5, 4 rows of 32 - 600 13.6 -> 7.7, 16 rows of
// 512 - 2048 20.7 -> 16.0; 4 tokens, one row of 1024 keys 14.9 -> 11.5, 4 rows of 32 - 600 13.8 -> 10.7.  Two or three groups
// of four warps per CTA were slower (4 tokens, one row: 13.4, 17.0): the merge through distributed shared memory grows.
// Semantics: nanovllm_jax/kv_cache.py:852-998 with query width > 1 (key p of row b is visible to token t when
// p < seq_lens[b] and, with positions given, p <= positions[b, t]).

#include "decode_cluster.cuh"

namespace nvj {

constexpr int kCwThreads = 128;
constexpr int kCwRowB = kD * 2;                  // one (token, KV head) row: 512 B
constexpr int kCwTokB = kHkv * kCwRowB;
constexpr int kCwPitch = kD + 4;                 // floats between output columns in the merge buffer: conflict-free stores
constexpr int kCwMaxWidth = 4;

template <int kTiles>
struct CwSmem {
  static constexpr int kCols = kTiles * 8;  // columns per KV head: token * 4 + head of the group, then padding
  union {
    struct {
      char q[kHkv][kCols][kCwRowB];  // [column][16-byte piece c of the row at c ^ (column & 7)]
      char k[kHkv][kBlk][kCwRowB];   // [key][piece c at c ^ (key & 7)]
      char v[kHkv][kBlk][kCwRowB];
    };
    float acc[kHkv * kCols][kCwPitch];
  };
  float2 ml[kHkv * kCols];
};

template <int kTiles>
__global__ void __launch_bounds__(kCwThreads, 3) decode_cluster_wide_kernel(DecodeParams p) {
  extern __shared__ __align__(128) unsigned char cw_smem_raw[];
  CwSmem<kTiles>& sm = *reinterpret_cast<CwSmem<kTiles>*>(cw_smem_raw);
  constexpr int kCols = CwSmem<kTiles>::kCols;
  using bf16 = __nv_bfloat16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int kvh = warp & 1, dh = warp >> 1;
  const int b = blockIdx.z, ctas = gridDim.x, cols = 4 * p.width;
  const int rank = ctas > 1 ? (int)cl_rank() : 0;

  pdl_wait();
  pdl_release();
  // ---- first trip: block ids of this CTA's first 32 blocks, the length, the tokens' positions, the queries
  const long long tbase = (long long)b * p.table_width;
  auto block_id = [&](int i) {
    const int jb = rank + i * ctas;
    return jb < p.table_width ? p.block_tables[tbase + jb] : -1;
  };
  int ids = block_id(lane);
  const int len = decode_row_len(p, b);
  int last[kTiles];  // last key that this lane's two columns of every tile may see (both are of one token)
#pragma unroll
  for (int n = 0; n < kTiles; ++n) {
    const int tok = n * 2 + (t >> 1);
    const int pos = tok < p.width ? (p.positions ? p.positions[(long long)b * p.width + tok] : 0x7fffffff) : -1;
    last[n] = pos < len - 1 ? pos : len - 1;
  }
  for (int i = threadIdx.x; i < kHkv * kCols * 32; i += kCwThreads) {  // 16-byte pieces
    const int h = i / (kCols * 32), col = (i >> 5) % kCols, piece = i & 31;
    uint4 x = make_uint4(0u, 0u, 0u, 0u);
    if (col < cols)
      x = ld_stream_u4(static_cast<const bf16*>(p.q) + (((long long)b * p.width + (col >> 2)) * kHq + h * kG + (col & 3)) * kD + piece * 8);
    *reinterpret_cast<uint4*>(sm.q[h][col] + ((piece ^ (col & 7)) << 4)) = x;
  }

  // ---- the CTA's blocks
  const int nb = (len + kBlk - 1) / kBlk;
  int asked = 0;
  auto next_id = [&]() -> long long {  // id of block rank + asked * ctas; -1 (and the flag) outside the pool
    if ((asked & 31) == 0 && asked > 0) ids = block_id(asked + lane);
    const long long blk = __shfl_sync(kFullMask, ids, asked & 31);
    if (blk >= 0 && blk < p.num_blocks) return blk;
    if (threadIdx.x == 0) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
    return -1;
  };
  const uint32_t k_at = smem_u32(sm.k[kvh]), v_at = smem_u32(sm.v[kvh]), q_at = smem_u32(sm.q[kvh]);
  // This warp's half (keys of parity dh) of one operand's 16 rows of block jb, as one group of copies.  Keys behind the last
  // one are read as that one again and masked below; a bad block is filled with zeros and masked.
  auto request = [&](uint32_t at, const char* cache, int jb, long long blk) {
    if (jb < nb) {
      const char* src = cache + (blk < 0 ? 0 : blk) * kBlk * kCwTokB + kvh * kCwRowB + lane * 16;
      const int end = len - 1 - jb * kBlk;
      const uint32_t size = blk < 0 ? 0u : 16u;
#pragma unroll
      for (int i = 0; i < kBlk / 2; ++i) {
        const int r = 2 * i + dh, rr = r < end ? r : (end < kBlk - 1 ? end : r);
        cl_copy16_or_zero(at + r * kCwRowB + ((lane ^ (r & 7)) << 4), src + rr * kCwTokB, size);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // (also an empty one: the waits count groups)
  };
  auto pair_sync = [&] { named_bar_sync(1 + kvh, 64); };  // the two warps of a KV head
  float o[8][kTiles][4];
  float m[kTiles][2], l[kTiles][2];
#pragma unroll
  for (int n = 0; n < kTiles; ++n) {
    m[n][0] = m[n][1] = kNegBig;
    l[n][0] = l[n][1] = 0.f;
#pragma unroll
    for (int d = 0; d < 8; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[d][n][e] = 0.f;
  }
  const float scale_log2 = p.scale * kLog2e;
  const uint32_t k_row = k_at + ((lane & 7) + ((lane >> 3) & 1) * 8) * kCwRowB, k_piece = lane >> 4;
  const uint32_t v_row = v_at + ((lane & 7) + (lane >> 4) * 8) * kCwRowB, v_piece = dh * 16 + ((lane >> 3) & 1);
  const uint32_t q_row = q_at + (lane & 7) * kCwRowB, q_piece = lane >> 3;  // four 16-byte pieces = two steps of 16 dims
  long long blk = rank < nb ? next_id() : -1;
  request(k_at, p.k_cache, rank, blk);
  request(v_at, p.v_cache, rank, blk);
  __syncthreads();  // Q is in place
  for (int j = rank; j < nb; j += ctas) {
    const bool good = blk >= 0;
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // this warp's K rows have landed
    pair_sync();
    float s[kTiles][4];
#pragma unroll
    for (int n = 0; n < kTiles; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
#pragma unroll
    for (int ks = 0; ks < 16; ks += 2) {
      uint32_t a0[4], a1[4];
      cm_ldsm4(k_row + (((ks * 2 + k_piece) ^ (lane & 7)) << 4), a0);
      cm_ldsm4(k_row + (((ks * 2 + 2 + k_piece) ^ (lane & 7)) << 4), a1);
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
        uint32_t qb[4];
        cm_ldsm4(q_row + n * 8 * kCwRowB + (((ks * 2 + q_piece) ^ (lane & 7)) << 4), qb);
        cm_mma<bf16>(s[n], a0, qb[0], qb[1]);
        cm_mma<bf16>(s[n], a1, qb[2], qb[3]);
      }
    }
    pair_sync();  // both warps have read the K rows
    const int jn = j + ctas;
    ++asked;
    blk = jn < nb ? next_id() : -1;
    request(k_at, p.k_cache, jn, blk);
    uint32_t hi[kTiles][2], lo[kTiles][2];  // the weights as B operands: [tile][keys 0-7 | 8-15]
    bool rescale = false;
    float alpha[kTiles][2];
#pragma unroll
    for (int n = 0; n < kTiles; ++n) {
      const int lim = good ? last[n] - j * kBlk : -1;  // keys of the block up to this one are visible
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = g + (e >> 1) * 8 <= lim ? s[n][e] * scale_log2 : kNegBig;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float mx = fmaxf(s[n][c], s[n][c + 2]);
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 4));
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 8));
        mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 16));
        const float mn = fmaxf(m[n][c], mx);
        alpha[n][c] = ex2_approx(m[n][c] - mn);
        rescale |= alpha[n][c] != 1.f;
        m[n][c] = mn;
        l[n][c] *= alpha[n][c];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = ex2_approx(s[n][e] - (m[n][e & 1] <= kNegBig ? 0.f : m[n][e & 1]));
      l[n][0] += s[n][0] + s[n][2];
      l[n][1] += s[n][1] + s[n][3];
#pragma unroll
      for (int k2 = 0; k2 < 2; ++k2) {
        hi[n][k2] = cm_transpose(cm_pack<bf16>(s[n][2 * k2], s[n][2 * k2 + 1], false));
        lo[n][k2] = cm_transpose(cm_pack<bf16>(s[n][2 * k2], s[n][2 * k2 + 1], true));
      }
    }
    if (__any_sync(kFullMask, rescale)) {
#pragma unroll
      for (int d = 0; d < 8; ++d)
#pragma unroll
        for (int n = 0; n < kTiles; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) o[d][n][e] *= alpha[n][e & 1];
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // this warp's V rows have landed
    pair_sync();
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      uint32_t a[4];
      cm_ldsm4_t(v_row + (((d * 2 + v_piece) ^ (lane & 7)) << 4), a);
#pragma unroll
      for (int n = 0; n < kTiles; ++n) {
        cm_mma<bf16>(o[d][n], a, hi[n][0], hi[n][1]);
        cm_mma<bf16>(o[d][n], a, lo[n][0], lo[n][1]);
      }
    }
    pair_sync();  // both warps have read the V rows
    request(v_at, p.v_cache, jn, blk);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();  // the merge buffer lies over the tiles

  // ---- this CTA's sums into shared memory, then the cluster's into the output
#pragma unroll
  for (int n = 0; n < kTiles; ++n)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      l[n][c] += __shfl_xor_sync(kFullMask, l[n][c], 4);
      l[n][c] += __shfl_xor_sync(kFullMask, l[n][c], 8);
      l[n][c] += __shfl_xor_sync(kFullMask, l[n][c], 16);
      const int col = kvh * kCols + n * 8 + 2 * t + c;
      if (dh == 0 && lane < 4) sm.ml[col] = make_float2(m[n][c], l[n][c]);
#pragma unroll
      for (int d = 0; d < 8; ++d) {
        sm.acc[col][dh * 128 + d * 16 + g] = o[d][n][c];
        sm.acc[col][dh * 128 + d * 16 + g + 8] = o[d][n][c + 2];
      }
    }
  if (ctas > 1) cl_sync(); else __syncthreads();
  // float4 pieces of [token][8 heads][256 dims], every CTA its share
  const int pieces = p.width * kHq * (kD / 4), per = (pieces + ctas - 1) / ctas;
  const int end = (rank + 1) * per < pieces ? (rank + 1) * per : pieces;
  float4* dst = reinterpret_cast<float4*>(p.out + (long long)b * p.width * kHq * kD);
  bool odd = false;
  for (int piece = rank * per + threadIdx.x; piece < end; piece += kCwThreads) {
    const int row = piece >> 6, tok = row / kHq, head = row - tok * kHq;
    const int col = (head / kG) * kCols + tok * 4 + (head % kG), d = (piece & 63) * 4;
    float M = kNegBig, L = 0.f;
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c0 = 0; c0 < ctas; c0 += 4) {  // four CTAs' pieces in flight
      float2 e[4];
      float4 x[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        e[c] = make_float2(kNegBig, 0.f);
        x[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c0 + c < ctas) {
          e[c] = ctas > 1 ? cl_ld2(cl_map(&sm.ml[col], c0 + c)) : sm.ml[col];
          x[c] = ctas > 1 ? cl_ld4(cl_map(&sm.acc[col][d], c0 + c)) : *reinterpret_cast<const float4*>(&sm.acc[col][d]);
        }
      }
      float mn = M;
#pragma unroll
      for (int c = 0; c < 4; ++c) mn = fmaxf(mn, e[c].x);
      const float a = ex2_approx(M - mn);
      M = mn;
      L *= a;
      y.x *= a; y.y *= a; y.z *= a; y.w *= a;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float f = ex2_approx(e[c].x - M);
        L = fmaf(e[c].y, f, L);
        y.x = fmaf(x[c].x, f, y.x); y.y = fmaf(x[c].y, f, y.y); y.z = fmaf(x[c].z, f, y.z); y.w = fmaf(x[c].w, f, y.w);
      }
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    y = make_float4(y.x * inv, y.y * inv, y.z * inv, y.w * inv);
    odd |= cl_not_finite(y);
    dst[piece] = y;
  }
  if (ctas > 1) cl_sync_read(odd);  // nobody leaves while its shared memory is being read
}

template <int kTiles>
static int launch_tiles(const DecodeParams& p, int cluster, cudaStream_t stream) {
  static PerDeviceFlags opted_in;
  return launch_clusters(decode_cluster_wide_kernel<kTiles>, opted_in, p, dim3(cluster), 1, kCwThreads, (int)sizeof(CwSmem<kTiles>), stream, p);
}

static bool cw_takes(const DecodeParams& p) {
  return p.width >= 2 && p.width <= kCwMaxWidth && p.batch <= kClMaxRows && !p.new_k && !p.packed_rows && !p.kv_indptr;
}
// Two CTAs at least where the mma.sync form is the alternative: it sums every other block of a row apart, one CTA all of them in a
// row, which is further from 64-bit attention (600 rows under 8 blocks, 2 tokens, plain / peaked / offset values: 1.84e-6 / 7.5e-7 / 4.1e-7 of
// the result's size with one CTA, 1.71e-6 / 6.5e-7 / 3.5e-7 with two, 1.70e-6 / 6.4e-7 / 3.5e-7 mma.sync; tcgen05, the alternative below
// that line, 2.1e-6 / 1.1e-6 / 3.5e-7 over 1000 rows under 12).  They cost 33 -> 38 us there (mma.sync 48).
static int cw_cluster(const DecodeParams& p, int sms) {
  const int c = cluster_size(p.batch, p.table_width, sms, 1, kCmPerSm, 8, kClMaxCluster);
  return c == 1 && p.table_width > 1 && wide_takes_mma_sync(p) ? 2 : c;
}

// Where the clusters serve the rows instead of tcgen05 (up to 4096 blocks of table with 2 tokens, 12288 with 3 and 4) or mma.sync
// (beyond, wide_takes_mma_sync).  First, few blocks per CTA (a block takes 0.7 us at 2 tokens, 0.9 at 3 and 4) and CTAs that are resident
// at once.  There tcgen05, which has clusters of its own, is as fast or faster by now, but further from 64-bit attention, so the lines
// stay where the clusters were ahead.  Clusters : tcgen05, rows of 1/4 - 1 and of 1/32 - 1/8 of the table (us, each launch behind a small kernel)
// and error relative to the result's size with plain, peaked and offset values:
//   2 tokens  16 x 128  19.1 : 16.5 and  9.7 :  9.4   1.8e-6 : 2.3e-6, 0.81e-6 : 1.7e-6, 2.0e-7 : 1.7e-7
//             64 x 40   18.8 : 19.3 and  9.5 : 10.1   1.8e-6 : 2.3e-6, 0.75e-6 : 2.0e-6, 2.3e-7 : 2.6e-7
//              2 x 157  12.9 :  9.8 and  7.5 :  8.8   1.9e-6 : 2.0e-6, 0.81e-6 : 0.73e-6, 2.3e-7 : 1.4e-7
//   3 tokens  32 x 64   21.3 : 18.0 and 12.0 : 10.3   1.8e-6 : 2.3e-6, 0.76e-6 : 1.8e-6, 2.0e-7 : 2.0e-7
//            128 x 16   19.9 : 25.1 and 10.6 : 17.7   1.7e-6 : 2.1e-6, 0.75e-6 : 1.3e-6, 2.8e-7 : 3.2e-7
//              4 x 128  17.9 : 11.5 and  9.1 :  9.1   1.8e-6 : 2.1e-6, 0.78e-6 : 0.80e-6, 2.1e-7 : 1.4e-7
//   4 tokens  64 x 40   23.8 : 21.5 and 13.3 : 11.8   1.8e-6 : 2.3e-6, 0.74e-6 : 1.9e-6, 2.3e-7 : 2.6e-7
//             16 x 32   16.6 : 10.7 and 13.8 :  9.5   1.6e-6 : 1.9e-6, 0.64e-6 : 0.76e-6, 1.9e-7 : 2.1e-7
// Beyond the line: 3 tokens, 16 x 128 (8 blocks per CTA, more CTAs than SMs) 22.9 : 17.6, 140 x 40 41.0 : 35.0; 2 tokens, 8 x 256 25.3 : 19.4; mma.sync,
// 50 x 96 30.6 : 30.1.
// Second, many short rows, of which every one costs the other forms a change of rows.  Rows of 1/4 - 1 and of 1/32 - 1/8 of the
// table; against tcgen05: 100 x 16 14.2 : 22.1 and 8.6 : 16.4 (2 tokens), 256 x 16 35.3 : 34.7 and 19.4 : 25.6 (3), 38.4 : 35.2 and
// 23.0 : 25.9 (4), 1000 x 12 72.4 : 92.8 and 34.6 : 68.5 (3), and closer to 64 bits.  Against mma.sync, 2 tokens: up to 24 blocks, which two CTAs share, 400 x
// 12 32.5 : 41.3 and 16.0 : 24.1, 2000 x 24 186.8 : 222.7 and 82.3 : 94.0, 4000 x 2 148 : 165 and 144 : 156, 16000 x 12 917 : 1151 and 572 : 674;
// from 25 on four CTAs, which only pay while they are few: 200 x 25 32.5 : 35.7 and 15.8 : 19.5, 400 x 25 56.9 : 56.8 and 29.5 : 29.3, 600 x
// 25 80.8 : 77.5 and 44.2 : 37.6, 2000 x 25 243 : 228 and 143 : 93.  3 and 4 tokens against mma.sync: ahead by 3 - 8% where the rows fill
// the table, behind by as much where they do not, 1000 x 16 95.2 : 101.5 and 52.3 : 53.0, 2000 x 8 132.6 : 140.9 and 96.8 : 92.5 (3 tokens),
// 150.7 : 155.9 and 115.8 : 105.4 (4), so they end at its line.
// Beyond 4 tokens a block takes 1.5 us and the tcgen05 form is the faster one from 4 blocks on.
bool decode_cluster_wide_pays(const DecodeParams& p) {
  const int sms = decode_wide_num_ctas();
  if (!cw_takes(p) || sms <= 0) return false;
  const int c = cw_cluster(p, sms), per_cta = (p.table_width + c - 1) / c;
  const long long ctas = (long long)c * p.batch;
  if (p.batch >= 100 && (p.width == 2 ? p.table_width <= (p.batch <= 400 ? 25 : 24) : p.table_width <= 16 && !wide_takes_mma_sync(p))) return true;
  if (p.width > 2 && per_cta == 8) return ctas <= sms;  // slower than tcgen05 there (4 x 128 above), at up to half its error
  return per_cta <= (p.width == 2 ? 12 : 7) && 100 * ctas <= (long long)kCmPerSm * sms;
}

// Rows of 2 - 4 bf16 query tokens over a dense table, already appended.
int launch_decode_cluster_wide(const DecodeParams& p, cudaStream_t stream) {
  if (!cw_takes(p)) return NVJ_ERR_UNSUPPORTED;
  const int sms = decode_wide_num_ctas();
  if (sms <= 0) return NVJ_ERR_LAUNCH;
  return p.width == 2 ? launch_tiles<1>(p, cw_cluster(p, sms), stream) : launch_tiles<2>(p, cw_cluster(p, sms), stream);
}

}  // namespace nvj
