// Paged GQA decode attention on thread-block clusters: the kernel for short batches, and for f32 / f16 caches, of the
// model's head layout (16-token blocks, 2 KV heads x 4 query heads, head_dim 256).
//
// A short batch is bound by latency, not by bytes.  The streaming kernel (paged_decode_wide.cu) needs 12 - 13 us for any:
// a scan that finds each CTA's range, block ids through shared memory, the first bulk copies, then a chain of fence,
// counter and fold through the far L2 for every row that is cut over CTAs.  Here the split needs no scan and the merge
// no counter:
//   * one cluster of C CTAs per (row, KV head); the cluster's warps take the row's blocks in turn (f32: units of 4 keys).
//     Block ids are requested together with the row's length (the table entry exists whatever the length is), so that K
//     and V are the second trip to memory;
//   * the warps merge through shared memory, the C CTAs through distributed shared memory: two cluster barriers instead
//     of fences and counters; rank r writes its 1 / C of the output;
//   * fused append: the cluster's first warp (f32: the one that the row's unit falls to) stores the new row, and whoever attends its key
//     reads it from the operand.
// Nothing waits on memory that somebody else must fill, so there is no wait to bound.
// Measured (us per launch, K/V cold, lengths spread over [n / 4, n]; the streaming kernel : this one): 4 rows of n = 512 tokens
// 10.6 : 5.5, 8 of 4096 19.1 : 13.2, 48 of 1024 19.1 : 16.5, 256 of 2048 108 : 106, 256 of 4096 204 : 200 (a first build, whose every
// copy selected its row, took 8% more).  f32: 8 rows of 64 - 512 tokens 221 (the generic kernel) : 7.4.
// Semantics: nanovllm_jax/kv_cache.py:852-998 for width-1 queries, nanovllm_jax/kernels/full_attention_triton.py:373-485
// for the fused append.

#include <type_traits>

#include "decode_cluster.cuh"
#include "row_argmax.cuh"

namespace nvj {

// ---- f32 caches (and f16 ones under f32 queries): fp32 products on the CUDA cores --------------------------------
// Every warp keeps a unit of 4 keys in flight in shared memory of its own (16-byte cp.async; the next unit's K rows are
// requested as soon as the scores are computed, its V rows after the weighted sum); lane l copies and later reads the same
// eight dims of every row, so this needs no barrier of any kind: 8 l .. 8 l + 7 of a 16-bit row, 4 l .. 4 l + 3 and
// 128 + 4 l .. of an f32 row.  (Every copy of a warp is then 512 bytes in a row.  With 8 l .. of an f32 row each copy took half of
// 32 sectors, and every sector crossed from the L2 twice.)  The 4 keys x 4 heads
// partial dot products are reduced by a select-free butterfly: lanes hold keys and heads in permuted order.
constexpr int kClWarps = 8;  // two CTAs per SM: a warp's chain of shuffles is long, four warps per scheduler overlap theirs
constexpr int kClThreads = kClWarps * 32;
constexpr int kClUnit = 4;  // keys a warp takes at a time

// The rows in flight [warp][K | V][key][row], later the merge buffers.
struct ClusterMerge {
  alignas(16) float acc[kClWarps][kG][kD];  // per warp; the merged sums of the CTA end up in acc[0]
  float2 ml[kClWarps][kG];                  // per warp (max, sum)
  float2 ML[kG];                            // of the CTA
};
template <typename T>
constexpr int cluster_smem_bytes() {
  constexpr int ring = kClWarps * 2 * kClUnit * kD * (int)sizeof(T);
  return ring > (int)sizeof(ClusterMerge) ? ring : (int)sizeof(ClusterMerge);
}

// Eight elements of a row per lane, as loaded.
template <typename T> struct ClRaw { uint4 v; };
template <> struct ClRaw<float> { uint4 v, w; };

// This lane's 16-byte pieces of a row: `at` is the lane's place in the ring's row, pieces 512 bytes apart.
__device__ __forceinline__ void cl_copy16(uint32_t dst, const char* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <typename T>
__device__ __forceinline__ void cl_copy_row(uint32_t row, const char* src, int lane) {
  cl_copy16(row + lane * 16, src + lane * 16);
  if constexpr (sizeof(T) == 4) cl_copy16(row + 512 + lane * 16, src + 512 + lane * 16);
}
__device__ __forceinline__ uint4 cl_lds(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
template <typename T>
__device__ __forceinline__ ClRaw<T> cl_read_row(uint32_t row, int lane) {
  ClRaw<T> r;
  r.v = cl_lds(row + lane * 16);
  if constexpr (sizeof(T) == 4) r.w = cl_lds(row + 512 + lane * 16);
  return r;
}
template <typename T>
__device__ __forceinline__ void cl_unpack(const ClRaw<T>& r, float2 (&o)[4]) {
  if constexpr (sizeof(T) == 4) {
    o[0] = make_float2(__uint_as_float(r.v.x), __uint_as_float(r.v.y));
    o[1] = make_float2(__uint_as_float(r.v.z), __uint_as_float(r.v.w));
    o[2] = make_float2(__uint_as_float(r.w.x), __uint_as_float(r.w.y));
    o[3] = make_float2(__uint_as_float(r.w.z), __uint_as_float(r.w.w));
  } else if constexpr (std::is_same<T, __half>::value) {
    o[0] = __half22float2(*reinterpret_cast<const __half2*>(&r.v.x));
    o[1] = __half22float2(*reinterpret_cast<const __half2*>(&r.v.y));
    o[2] = __half22float2(*reinterpret_cast<const __half2*>(&r.v.z));
    o[3] = __half22float2(*reinterpret_cast<const __half2*>(&r.v.w));
  } else {
    o[0] = bf16x2_to_float2(r.v.x);
    o[1] = bf16x2_to_float2(r.v.y);
    o[2] = bf16x2_to_float2(r.v.z);
    o[3] = bf16x2_to_float2(r.v.w);
  }
}

// A launch that runs beside the kernel in front of it ends after that kernel: one CTA holds the grid open, and then clears the
// word that told the CTAs to go ahead (whoever has not read it yet waits for the kernel in front, which has ended by now).
__device__ __forceinline__ void cl_end_beside(const DecodeParams& p) {
  if (p.beside && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    pdl_wait();
    if (threadIdx.x == 0) st_release_gpu(p.beside, 0);
  }
}
// The CTAs' sums [head][pitch] and (max, sum) pairs, at the same places in every CTA of the cluster, into the output: rank
// r takes its 1 / ctas of the float4 pieces of [heads][256 dims].  Returns what cl_sync_read() asks for.
// `store` gets a piece's index and its four values; `base`: the cluster's rank of the first of these CTAs.
template <int kHeads, class Store>
__device__ __forceinline__ bool cl_fold_cluster(const float* acc, int pitch, const float2* ML, int ctas, int rank, int base, int threads,
                                                Store store) {
  constexpr int kPieces = kHeads * kD / 4;
  const int per = (kPieces + ctas - 1) / ctas;
  bool odd = false;
  for (int i = threadIdx.x; i < per; i += threads) {
    const int piece = rank * per + i, h = piece >> 6, d = (piece & 63) * 4;
    if (piece >= kPieces) break;
    float2 e[kClMaxCluster];
    float4 x[kClMaxCluster];
#pragma unroll
    for (int c = 0; c < kClMaxCluster; ++c) {
      if (c % 4 == 0 && c >= ctas) break;  // (four at a time; all sixteen always: six layers of 200 rows of 64 - 512 keys 174.5 us, so 170.4)
      e[c] = make_float2(kNegBig, 0.f);
      x[c] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < ctas) {
        e[c] = cl_ld2(cl_map(ML + h, base + c));
        x[c] = cl_ld4(cl_map(acc + h * pitch + d, base + c));
      }
    }
    float M = kNegBig, L = 0.f;
#pragma unroll
    for (int c = 0; c < kClMaxCluster; ++c) {
      if (c % 4 == 0 && c >= ctas) break;
      M = fmaxf(M, e[c].x);
    }
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int c = 0; c < kClMaxCluster; ++c) {
      if (c % 4 == 0 && c >= ctas) break;
      const float f = ex2_approx(e[c].x - M);
      L = fmaf(e[c].y, f, L);
      y.x = fmaf(x[c].x, f, y.x); y.y = fmaf(x[c].y, f, y.y); y.z = fmaf(x[c].z, f, y.z); y.w = fmaf(x[c].w, f, y.w);
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    y = make_float4(y.x * inv, y.y * inv, y.z * inv, y.w * inv);
    odd |= cl_not_finite(y);
    store(piece, y);
  }
  return odd;
}

template <typename T>
__global__ void __launch_bounds__(kClThreads, 2) decode_cluster_kernel(DecodeParams p) {
  extern __shared__ __align__(128) unsigned char cl_smem_raw[];
  ClusterMerge& sm = *reinterpret_cast<ClusterMerge*>(cl_smem_raw);
  constexpr int kRowB = kD * (int)sizeof(T), kTokB = kHkv * kRowB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z, kvh = blockIdx.y, ctas = gridDim.x;
  const uint32_t rank = ctas > 1 ? cl_rank() : 0u;
  const int first = (int)rank * kClWarps + warp, stride = ctas * kClWarps;  // this warp's units: first, first + stride, ...

  pdl_wait();
  pdl_release();
  // ---- first trip: the ids of this warp's first 32 units, the length, the query
  const long long tbase = decode_table_base(p, b);
  int pages = p.table_width;
  if (p.kv_indptr) pages = p.kv_indptr[b + 1] - (int)tbase;
  auto unit_id = [&](int i) {  // lane i of a batch: block id of unit i
    const int jb = (first + i * stride) / (kBlk / kClUnit);
    return jb < pages ? p.block_tables[tbase + jb] : -1;
  };
  int ids = unit_id(lane);
  const int len = decode_row_len(p, b);  // the same in every thread of the cluster
  const long long qi = decode_query_index(p, b);
  if (p.packed_rows && p.query_start_loc[b + 1] - p.query_start_loc[b] != 1) return;  // not this pass's row (the whole cluster leaves)
  constexpr bool kFull = sizeof(T) == 4;
  const int d0 = lane * (kFull ? 4 : 8), d1 = kFull ? kD / 2 + lane * 4 : lane * 8 + 4;  // this lane's dims: four from each
  // query heads in slot order (slot h of a lane holds head h ^ hperm), times scale * log2(e)
  const int rperm = lane >> 3, h_own = (lane >> 1) & 3;
  float2 q2[kG][4];
#pragma unroll
  for (int h = 0; h < kG; ++h) {
    const long long off = (qi * kHq + kvh * kG + (h ^ h_own)) * kD;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const long long at = off + (i ? d1 : d0);
      if (p.q_dtype == NVJ_F32) {
        const float4 x = *reinterpret_cast<const float4*>(static_cast<const float*>(p.q) + at);
        q2[h][2 * i] = make_float2(x.x, x.y); q2[h][2 * i + 1] = make_float2(x.z, x.w);
      } else {
        const uint2 x = *reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p.q) + at);
        if (p.q_dtype == NVJ_BF16) {
          q2[h][2 * i] = bf16x2_to_float2(x.x); q2[h][2 * i + 1] = bf16x2_to_float2(x.y);
        } else {
          q2[h][2 * i] = __half22float2(*reinterpret_cast<const __half2*>(&x.x));
          q2[h][2 * i + 1] = __half22float2(*reinterpret_cast<const __half2*>(&x.y));
        }
      }
    }
    const float c = p.scale * kLog2e;
#pragma unroll
    for (int i = 0; i < 4; ++i) { q2[h][i].x *= c; q2[h][i].y *= c; }
  }

  // ---- fused append: where the new row goes; its key (if attended) is read from the operand.  The warp that the row's unit falls to
  // stores it: it has the block's id among its own.  (With the warp of unit 0, which has to fetch it, every warp waits for one trip more:
  // f32, 8 rows of 64 - 512 keys 7.7 us : 7.6, 32 of 1000 - 2000 41.6 : 41.3.)
  int new_key = -1;
  const char* new_k = nullptr;
  const char* new_v = nullptr;
  if (p.new_k && len > 0) {
    const int pos = p.pre_append ? p.seq_lens[b] : p.positions[b];
    new_k = static_cast<const char*>(p.new_k) + (long long)b * kTokB + kvh * kRowB;
    new_v = static_cast<const char*>(p.new_v) + (long long)b * kTokB + kvh * kRowB;
    const int jt = pos / kBlk, unit = pos / kClUnit, turn = (unit - first) / stride;
    if (pos < 0 ? first == 0 : unit % stride == first) {
      const int held = __shfl_sync(kFullMask, ids, turn & 31);
      const long long tgt = pos < 0 || jt >= p.table_width ? -1 : !p.kv_indptr && turn < 32 ? held : p.block_tables[tbase + jt];
      if (tgt >= 0 && tgt < p.num_blocks) {
        if (pos < len) new_key = pos;
        const long long dst = (tgt * kBlk + pos % kBlk) * kTokB + kvh * kRowB;
#pragma unroll
        for (int i = 0; i < (int)sizeof(T) / 2; ++i) {
          const int o = (i * 32 + lane) * 16;
          *reinterpret_cast<uint4*>(const_cast<char*>(p.k_cache) + dst + o) = *reinterpret_cast<const uint4*>(new_k + o);
          *reinterpret_cast<uint4*>(const_cast<char*>(p.v_cache) + dst + o) = *reinterpret_cast<const uint4*>(new_v + o);
        }
      } else if (lane == 0) {
        atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
      }
    }
  }

  // ---- the warp's units: four keys at a time, key slot r of a lane holds key r ^ rperm of the unit
  const int units = (len + kClUnit - 1) / kClUnit;
  float2 acc[kG][4];
  float m4[kG], m_own = kNegBig, l_part = 0.f;
#pragma unroll
  for (int h = 0; h < kG; ++h) {
    m4[h] = kNegBig;
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[h][i] = make_float2(0.f, 0.f);
  }
  // Row of key `key` of unit u, from the cache or (the step's own key) from the operand.  Keys behind the last attended one
  // are read as that one again and masked below: no load depends on a branch, so all of a unit's loads go out together.
  auto row_of = [&](const char* cache, const char* fresh, int u, long long blk, int key) -> const char* {
    int t = u * kClUnit + key;
    t = t < len ? t : len - 1;
    const char* row = cache + (blk * kBlk + t % kBlk) * kTokB + kvh * kRowB;
    return t == new_key ? fresh : row;
  };
  const uint32_t k_at = smem_u32(cl_smem_raw) + warp * (2 * kClUnit * kRowB), v_at = k_at + kClUnit * kRowB;
  // the unit's rows of one operand, as one group of copies (also an empty one: the waits count groups)
  auto request = [&](uint32_t at, const char* cache, const char* fresh, int u, long long blk) {
    if (u < units) {
#pragma unroll
      for (int r = 0; r < kClUnit; ++r) cl_copy_row<T>(at + r * kRowB, row_of(cache, fresh, u, blk, r), lane);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // The warp's i-th unit that lies in the pool, at or after unit u; a bad block id is flagged and its keys are left out.
  int u = first, i = 0;
  auto next_unit = [&](int& u, int& i) -> long long {
    for (; u < units; u += stride, ++i) {
      if ((i & 31) == 0 && i > 0) ids = unit_id(i + lane);
      const long long blk = __shfl_sync(kFullMask, ids, i & 31);
      if (blk >= 0 && blk < p.num_blocks) return blk;
      if (lane == 0) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
    }
    return 0;
  };
  long long blk = next_unit(u, i);
  request(k_at, p.k_cache, new_k, u, blk);
  request(v_at, p.v_cache, new_v, u, blk);
  while (u < units) {
    const int left = len - u * kClUnit;  // keys of the unit that are attended (at least one)
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // K has landed
    float s[16];
#pragma unroll
    for (int r = 0; r < kClUnit; ++r) {  // key slot r of a lane holds key r ^ rperm of the unit
      float2 k2[4];
      cl_unpack(cl_read_row<T>(k_at + (r ^ rperm) * kRowB, lane), k2);
#pragma unroll
      for (int h = 0; h < kG; ++h) {
        float2 a = fma2(q2[h][0], k2[0], make_float2(0.f, 0.f));
        a = fma2(q2[h][1], k2[1], a);
        a = fma2(q2[h][2], k2[2], a);
        a = fma2(q2[h][3], k2[3], a);
        s[r * 4 + h] = a.x + a.y;
      }
    }
    u += stride;
    ++i;
    blk = next_unit(u, i);
    request(k_at, p.k_cache, new_k, u, blk);
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] += __shfl_xor_sync(kFullMask, s[e + 8], 16);
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] += __shfl_xor_sync(kFullMask, s[e + 4], 8);
#pragma unroll
    for (int e = 0; e < 2; ++e) s[e] += __shfl_xor_sync(kFullMask, s[e + 2], 4);
    s[0] += __shfl_xor_sync(kFullMask, s[1], 2);
    float sc = s[0] + __shfl_xor_sync(kFullMask, s[0], 1);  // score of (key rperm, head h_own)
    if (rperm >= left) sc = -INFINITY;
    float bm = fmaxf(sc, __shfl_xor_sync(kFullMask, sc, 8));
    bm = fmaxf(bm, __shfl_xor_sync(kFullMask, bm, 16));
    if (__any_sync(kFullMask, bm > m_own)) {
#pragma unroll
      for (int j = 0; j < kG; ++j) {
        const float bj = __shfl_sync(kFullMask, bm, j * 2);
        const float mn = fmaxf(m4[j], bj);
        const float a = ex2_approx(m4[j] - mn);
        m4[j] = mn;
#pragma unroll
        for (int c = 0; c < 4; ++c) { acc[j][c].x *= a; acc[j][c].y *= a; }
        if (h_own == j) { l_part *= a; m_own = mn; }
      }
    }
    const float pw = ex2_approx(sc - m_own);
    l_part += pw;
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // V has landed
#pragma unroll
    for (int r = 0; r < kClUnit; ++r) {
      float2 v2[4];
      cl_unpack(cl_read_row<T>(v_at + r * kRowB, lane), v2);
#pragma unroll
      for (int h = 0; h < kG; ++h) {
        const float w = __shfl_sync(kFullMask, pw, r * 8 + h * 2);
        const float2 ww = make_float2(w, w);
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[h][c] = fma2(ww, v2[c], acc[h][c]);
      }
    }
    request(v_at, p.v_cache, new_v, u, blk);  // (this lane alone reads what it copied)
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();  // the merge buffers lie over the rings

  // ---- merge the eight warps, then the cluster
  float lh = l_part;
  lh += __shfl_xor_sync(kFullMask, lh, 8);
  lh += __shfl_xor_sync(kFullMask, lh, 16);
#pragma unroll
  for (int h = 0; h < kG; ++h) {
    const float l = __shfl_sync(kFullMask, lh, h * 2);
    if (lane == 0) sm.ml[warp][h] = make_float2(m4[h], l);
    *reinterpret_cast<float4*>(&sm.acc[warp][h][d0]) = make_float4(acc[h][0].x, acc[h][0].y, acc[h][1].x, acc[h][1].y);
    *reinterpret_cast<float4*>(&sm.acc[warp][h][d1]) = make_float4(acc[h][2].x, acc[h][2].y, acc[h][3].x, acc[h][3].y);
  }
  __syncthreads();
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  float M = kNegBig, L = 0.f;
  static_assert(kClThreads == kG * kD / 4, "a thread merges four dims of one head");
  const int h = threadIdx.x / (kD / 4), d4 = (threadIdx.x % (kD / 4)) * 4;
#pragma unroll
  for (int w = 0; w < kClWarps; ++w) M = fmaxf(M, sm.ml[w][h].x);
#pragma unroll
  for (int w = 0; w < kClWarps; ++w) {
    const float2 e = sm.ml[w][h];
    const float f = ex2_approx(e.x - M);
    const float4 x = *reinterpret_cast<const float4*>(&sm.acc[w][h][d4]);
    L = fmaf(e.y, f, L);
    o.x = fmaf(x.x, f, o.x); o.y = fmaf(x.y, f, o.y); o.z = fmaf(x.z, f, o.z); o.w = fmaf(x.w, f, o.w);
  }
  float* dst = p.out + (qi * kHq + kvh * kG) * kD;
  if (ctas == 1) {
    const float inv = L > 0.f ? 1.f / L : 0.f;
    reinterpret_cast<float4*>(dst)[threadIdx.x] = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
    return;
  }
  __syncthreads();  // acc[0] is overwritten
  *reinterpret_cast<float4*>(&sm.acc[0][h][d4]) = o;
  if (d4 == 0) sm.ML[h] = make_float2(M, L);
  cl_sync();
  const bool odd = cl_fold_cluster<kG>(&sm.acc[0][0][0], kD, sm.ML, ctas, (int)rank, 0, kClThreads,
                                       [&](int piece, float4 y) { reinterpret_cast<float4*>(dst)[piece] = y; });
  cl_sync_read(odd);  // nobody leaves while its shared memory is being read
}

// ---- 16-bit caches: the products on tensor-core tiles -------------------------------------------------------------
// A warp's unit is a whole block (16 keys) of its KV head.  Both products are taken transposed, so that the four query
// heads sit in the N = 8 columns of mma.m16n8k16 instead of wasting 12 of 16 rows:
//   S^T = K Q^T   M = 16 keys, N = 8 columns (the four heads, twice), 16 steps over the dims;
//   O^T = V^T P^T  M = 16 dims (16 tiles), N = 8: columns 0-3 take the weights rounded to 16 bits, columns 4-7 what the
//                 rounding left over, so that one MMA carries both terms; they are added at the end.
// 32 MMAs and 32 ldmatrix per block and head, an eighth of the instructions of the CUDA-core form above, which bound
// that form at ~1500 cycles per unit of 4 keys and warp.  One block per warp is in flight: the next block's K rows are
// requested as soon as the scores are computed, its V rows after the weighted sum, and three CTAs of 64 KiB overlap on an
// SM.  (Three blocks per warp and one CTA per SM were measured: the same within 5% where CTAs are few, worse where they
// are many.  What one SM takes in, ~57 GB/s, is the limit then, so a row's blocks must be spread over SMs instead.)
constexpr int kCmWarps = 4;
constexpr int kCmThreads = kCmWarps * 32;
constexpr int kCmPitch = kD + 4;  // floats between the columns of a warp's output tile: conflict-free stores

struct CmSmem {
  union {
    char ring[kCmWarps][2][kBlk][kD * 2];  // [warp][K | V][key][16-byte piece c of the row at c ^ (key & 7)]
    struct {
      float acc[kCmWarps * kG][kCmPitch];  // [warp, head][dim]; the CTA's merged sums end up in the first rows, one per head
      float2 ml[kCmWarps][kG];
      float2 ML[kHq];
    } m;
  };
  float2 pick[kClMaxCluster];  // in the cluster's first CTA: every CTA's best output value and (as bits) its index
  float2 pick_warp[kCmWarps];
};

// Ahead of pdl_wait(), while the append in front is at work and memory is idle: K and V rows of block jb, the first that this warp
// will walk, on their way into the L2.  What is read here may be about to change, so it is a hint and nothing else: relaxed loads
// (they leave no line in the L1 that a load behind the wait could find), an id that is checked against the pool, a prefetch.
// Measured, six layers of norm + RoPE + append and this: 48 rows of 128 - 2048 keys 164.2 -> 154.3 us, 200 of 64 - 512 186 -> 174, 256 of
// 1024 - 4096 1254 -> 1247; with the two first blocks 164.9, and with the append letting its dependents go before its own wait 163.5
// (both take bandwidth from the kernel that still runs).  Only where the rows have been appended by a launch of their own: in front
// of a fused append may be anything, and where that has long ended the extra trip to memory is lost (64 rows from host memory 512.8 ->
// 517.2); and only in CTAs that start together (256 rows, fused, 1674 -> 1683).
__device__ __forceinline__ void cm_prefetch_block(const DecodeParams& p, int b, int kvh, int jb, int lane) {
  if ((int)((blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x) >= p.early_ctas || jb >= p.table_width) return;
  const int len = ld_relaxed_gpu(p.seq_lens + b), blk = ld_relaxed_gpu(p.block_tables + (long long)b * p.table_width + jb);
  if (len <= jb * kBlk || blk < 0 || blk >= p.num_blocks) return;
  const char* cache = lane < kBlk ? p.k_cache : p.v_cache;
  l2_prefetch(cache + ((long long)blk * kBlk + (lane & (kBlk - 1))) * kTokenBytes + kvh * kRowBytes, kRowBytes);
}

// kPick: the token pick of a decode step (DecodeParams::pick_tokens).  All CTAs of a row then form one cluster, also where
// they take a KV head each.
template <typename T, bool kBoth, bool kPick>
__global__ void __launch_bounds__(kCmThreads, 3) decode_cluster_mma_kernel(DecodeParams p) {
  extern __shared__ __align__(128) unsigned char cl_smem_raw[];
  CmSmem& sm = *reinterpret_cast<CmSmem*>(cl_smem_raw);
  constexpr int kRowB = kD * 2, kTokB = kHkv * kRowB;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int b = blockIdx.z, kvh = kBoth ? warp & 1 : blockIdx.y, ctas = gridDim.x;
  const int rank = blockIdx.x;  // among the CTAs that share the head's (or both heads') blocks
  constexpr int kWalkers = kBoth ? kCmWarps / 2 : kCmWarps;  // warps of the CTA that share a KV head's blocks
  const int first = rank * kWalkers + (kBoth ? warp >> 1 : warp), stride = ctas * kWalkers;  // this warp's blocks: first, first + stride, ...

  cm_prefetch_block(p, b, kvh, first, lane);
  if (!p.beside || ld_acquire_gpu(p.beside) == 0) pdl_wait();
  pdl_release();
  // ---- first trip: the ids of this warp's first 32 blocks, the length, the query
  const long long tbase = decode_table_base(p, b);
  int pages = p.table_width;
  if (p.kv_indptr) pages = p.kv_indptr[b + 1] - (int)tbase;
  auto block_id = [&](int i) {
    const int jb = first + i * stride;
    return jb < pages ? p.block_tables[tbase + jb] : -1;
  };
  int ids = block_id(lane);
  const int len = decode_row_len(p, b);
  const long long qi = decode_query_index(p, b);
  if (p.packed_rows && p.query_start_loc[b + 1] - p.query_start_loc[b] != 1) {  // not this pass's row (the whole cluster leaves)
    cl_end_beside(p);
    return;
  }
  uint32_t qb[16][2];  // Q^T as the B operand: column g = head g & 3
  {
    const char* q = static_cast<const char*>(p.q) + ((qi * kHq + kvh * kG + (g & 3)) * kD) * 2;
#pragma unroll
    for (int ks = 0; ks < 16; ++ks) {
      qb[ks][0] = *reinterpret_cast<const uint32_t*>(q + ks * 32 + t * 4);
      qb[ks][1] = *reinterpret_cast<const uint32_t*>(q + ks * 32 + 16 + t * 4);
    }
  }

  // ---- fused append: where the new row goes; its key (if attended) is read from the operand.  The row's first warp stores it, not the
  // one that its block falls to, which has the id but also the longest walk: eight steps of a graph, stored by that one : by the first,
  // 39 rows of 200 - 800 keys 129.9 us : 115.7, 40 of 700 - 2800 276.5 : 267.1, 256 of 200 - 800 468.5 : 459.9; one launch, 16 rows of 500 -
  // 2000 10.7 : 10.2, 150 of 512 - 1024 45.3 : 45.1.
  int new_key = -1;
  const char* new_k = nullptr;
  const char* new_v = nullptr;
  if (p.new_k && len > 0) {
    const int pos = p.pre_append ? p.seq_lens[b] : p.positions[b];
    new_k = static_cast<const char*>(p.new_k) + (long long)b * kTokB + kvh * kRowB + lane * 16;
    new_v = static_cast<const char*>(p.new_v) + (long long)b * kTokB + kvh * kRowB + lane * 16;
    if (pos >= 0) {
      const int jt = pos / kBlk;
      const long long tgt = jt < p.table_width ? (long long)p.block_tables[tbase + jt] : -1;
      if (tgt >= 0 && tgt < p.num_blocks) {
        if (pos < len) new_key = pos;
        if (first == 0) {
          const long long dst = (tgt * kBlk + pos % kBlk) * kTokB + kvh * kRowB + lane * 16;
          *reinterpret_cast<uint4*>(const_cast<char*>(p.k_cache) + dst) = *reinterpret_cast<const uint4*>(new_k);
          *reinterpret_cast<uint4*>(const_cast<char*>(p.v_cache) + dst) = *reinterpret_cast<const uint4*>(new_v);
        }
      } else if (first == 0 && lane == 0) {
        atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
      }
    } else if (!std::is_same<T, __nv_bfloat16>::value && first == 0 && lane == 0) {
      atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
    }
  }

  // ---- the warp's blocks
  const int nb = (len + kBlk - 1) / kBlk;
  int asked = 0;  // blocks requested so far
  auto next_id = [&]() -> long long {  // id of block first + asked * stride; -1 (and the flag) outside the pool
    if ((asked & 31) == 0 && asked > 0) ids = block_id(asked + lane);
    const long long blk = __shfl_sync(kFullMask, ids, asked & 31);
    if (blk >= 0 && blk < p.num_blocks) return blk;
    if (lane == 0) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
    return -1;
  };
  const uint32_t k_at = smem_u32(sm.ring[warp][0]), v_at = smem_u32(sm.ring[warp][1]);
  // The 16 rows of block jb of one operand into `at`, as one group of copies.  Keys behind the last attended one are read as
  // that one again and masked below; a bad block is filled with zeros and masked.
  auto request = [&](uint32_t at, const char* cache, const char* fresh, int jb, long long blk) {
    if (jb < nb) {
      const char* src = cache + (blk < 0 ? 0 : blk) * kBlk * kTokB + kvh * kRowB + lane * 16;
      const int last = len - 1 - jb * kBlk, mine = new_key - jb * kBlk;
      if (blk >= 0 && last >= kBlk - 1 && (unsigned)mine >= (unsigned)kBlk) {  // a whole block as it lies in the cache: constant offsets
#pragma unroll
        for (int r = 0; r < kBlk; ++r) cl_copy16(at + r * kRowB + ((lane ^ (r & 7)) << 4), src + r * kTokB);
      } else {
        const uint32_t size = blk < 0 ? 0u : 16u;
#pragma unroll 8
        for (int r = 0; r < kBlk; ++r) {
          const int rr = r < last ? r : (last < kBlk - 1 ? last : r);
          cl_copy16_or_zero(at + r * kRowB + ((lane ^ (r & 7)) << 4), rr == mine ? fresh : src + rr * kTokB, size);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // (also an empty one: the waits count groups)
  };
  float o[16][4];
#pragma unroll
  for (int n = 0; n < 16; ++n)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
  float m[2] = {kNegBig, kNegBig}, l[2] = {0.f, 0.f};  // of heads (2 t) & 3, (2 t + 1) & 3
  const float scale_log2 = p.scale * kLog2e;
  const uint32_t k_row = k_at + ((lane & 7) + ((lane >> 3) & 1) * 8) * kRowB, k_piece = lane >> 4;
  const uint32_t v_row = v_at + ((lane & 7) + (lane >> 4) * 8) * kRowB, v_piece = (lane >> 3) & 1;
  long long blk = first < nb ? next_id() : -1;
  request(k_at, p.k_cache, new_k, first, blk);
  request(v_at, p.v_cache, new_v, first, blk);
  for (int j = first; j < nb; j += stride) {
    const int left = blk >= 0 ? len - j * kBlk : 0;  // keys of the block that are attended
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // K has landed
    __syncwarp();
    float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};  // two chains of eight
#pragma unroll
    for (int ks = 0; ks < 16; ks += 2) {
      uint32_t a[4];
      cm_ldsm4(k_row + (((ks * 2 + k_piece) ^ (lane & 7)) << 4), a);
      cm_mma<T>(s0, a, qb[ks][0], qb[ks][1]);
      cm_ldsm4(k_row + (((ks * 2 + 2 + k_piece) ^ (lane & 7)) << 4), a);
      cm_mma<T>(s1, a, qb[ks + 1][0], qb[ks + 1][1]);
    }
    __syncwarp();
    const int jn = j + stride;
    ++asked;
    blk = jn < nb ? next_id() : -1;
    request(k_at, p.k_cache, new_k, jn, blk);
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = g + (e >> 1) * 8 < left ? (s0[e] + s1[e]) * scale_log2 : kNegBig;
    float alpha[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      float mx = fmaxf(s[c], s[c + 2]);
      mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 4));
      mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 8));
      mx = fmaxf(mx, __shfl_xor_sync(kFullMask, mx, 16));
      const float mn = fmaxf(m[c], mx);
      alpha[c] = ex2_approx(m[c] - mn);
      m[c] = mn;
      l[c] *= alpha[c];
    }
    if (__any_sync(kFullMask, alpha[0] != 1.f || alpha[1] != 1.f)) {
#pragma unroll
      for (int n = 0; n < 16; ++n) {
        o[n][0] *= alpha[0]; o[n][1] *= alpha[1];
        o[n][2] *= alpha[0]; o[n][3] *= alpha[1];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = ex2_approx(s[e] - (m[e & 1] <= kNegBig ? 0.f : m[e & 1]));  // nothing attended yet: 0
    l[0] += s[0] + s[2];
    l[1] += s[1] + s[3];
    const uint32_t b0 = cm_transpose(cm_pack<T>(s[0], s[1], t >= 2)), b1 = cm_transpose(cm_pack<T>(s[2], s[3], t >= 2));
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // V has landed
    __syncwarp();
#pragma unroll
    for (int n = 0; n < 16; ++n) {
      uint32_t a[4];
      cm_ldsm4_t(v_row + (((n * 2 + v_piece) ^ (lane & 7)) << 4), a);
      cm_mma<T>(o[n], a, b0, b1);
    }
    __syncwarp();
    request(v_at, p.v_cache, new_v, jn, blk);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();  // the merge buffers lie over the rings

  // ---- merge the warps, then the cluster
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    l[c] += __shfl_xor_sync(kFullMask, l[c], 4);
    l[c] += __shfl_xor_sync(kFullMask, l[c], 8);
    l[c] += __shfl_xor_sync(kFullMask, l[c], 16);
    if (lane < 2) sm.m.ml[warp][2 * t + c] = make_float2(m[c], l[c]);
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)  // both terms of a column are added: of two tiles a lane keeps one and gives the other away
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float keep = t < 2 ? o[2 * k][e] : o[2 * k + 1][e], give = t < 2 ? o[2 * k + 1][e] : o[2 * k][e];
      sm.m.acc[warp * kG + 2 * (t & 1) + (e & 1)][(2 * k + (t >> 1)) * 16 + g + 8 * (e >> 1)] = keep + __shfl_xor_sync(kFullMask, give, 2);
    }
  __syncthreads();
  constexpr int kHeads = kBoth ? kHq : kG;
  constexpr int kPieces = kHeads * kD / 4, kPer = kPieces / kCmThreads;  // float4 pieces of the output, and per thread
  float* dst = p.out + (qi * kHq + (kBoth ? 0 : kvh * kG)) * kD;
  ArgBest best;
  auto store = [&](int piece, float4 y) {
    reinterpret_cast<float4*>(dst)[piece] = y;
    if constexpr (kPick) {
      const int i = (kBoth ? 0 : kvh * kG * kD) + piece * 4;
      best.take(y.x, i); best.take(y.y, i + 1); best.take(y.z, i + 2); best.take(y.w, i + 3);
    }
  };
  float4 sum[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const int piece = k * kCmThreads + threadIdx.x, head = piece >> 6, h = head & (kG - 1), d4 = (piece & 63) * 4;
    constexpr int kStep = kCmWarps / kWalkers;
    const int w0 = kBoth ? head / kG : 0;  // the first warp of this head
    float M = kNegBig, L = 0.f;
#pragma unroll
    for (int w = 0; w < kWalkers; ++w) M = fmaxf(M, sm.m.ml[w0 + w * kStep][h].x);
    sum[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int w = 0; w < kWalkers; ++w) {
      const float2 e = sm.m.ml[w0 + w * kStep][h];
      const float f = ex2_approx(e.x - M);
      const float4 x = *reinterpret_cast<const float4*>(&sm.m.acc[(w0 + w * kStep) * kG + h][d4]);
      L = fmaf(e.y, f, L);
      sum[k].x = fmaf(x.x, f, sum[k].x); sum[k].y = fmaf(x.y, f, sum[k].y);
      sum[k].z = fmaf(x.z, f, sum[k].z); sum[k].w = fmaf(x.w, f, sum[k].w);
    }
    if (ctas == 1) {
      const float inv = L > 0.f ? 1.f / L : 0.f;
      store(piece, make_float4(sum[k].x * inv, sum[k].y * inv, sum[k].z * inv, sum[k].w * inv));
    } else if ((piece & 63) == 0) {
      sm.m.ML[head] = make_float2(M, L);
    }
  }
  bool odd = false;
  if (ctas > 1) {
    __syncthreads();  // the first rows are overwritten
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int piece = k * kCmThreads + threadIdx.x;
      *reinterpret_cast<float4*>(&sm.m.acc[piece >> 6][(piece & 63) * 4]) = sum[k];
    }
    cl_sync();
    odd = cl_fold_cluster<kHeads>(&sm.m.acc[0][0], kCmPitch, sm.m.ML, ctas, rank, kPick && !kBoth ? kvh * ctas : 0, kCmThreads, store);
  }
  const int members = kPick && !kBoth ? kHkv * ctas : ctas;  // CTAs of the cluster
  if constexpr (kPick) {
    if (members > 1 && ctas == 1) cl_sync();  // (no barrier so far: the cluster's first CTA has to have started)
    best.reduce_warp();
    if (lane == 0) sm.pick_warp[warp] = make_float2(best.v, __int_as_float(best.i));
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
      for (int w = 1; w < kCmWarps; ++w) best.take(sm.pick_warp[w].x, __float_as_int(sm.pick_warp[w].y));
      if (members > 1) cl_st2(cl_map(&sm.pick[kBoth ? rank : kvh * ctas + rank], 0), best.v, best.i);
    }
  }
  // nobody leaves while its shared memory is being read; every candidate has arrived
  if (members > 1) {
    if constexpr (kPick) cl_sync();
    else cl_sync_read(odd);
  }
  if constexpr (kPick) {
    if (threadIdx.x == 0 && rank == 0 && (kBoth || kvh == 0)) {
      for (int c = 1; c < members; ++c) best.take(sm.pick[c].x, __float_as_int(sm.pick[c].y));
      p.pick_tokens[b] = best.index();
      advance_row(p.pick_lens, p.pick_positions, b, (long long)p.table_width * p.block_size, p.status);  // (all of the row's CTAs have read it)
    }
  }
  cl_end_beside(p);
}

// The tensor-core form's launch for a batch: CTAs per cluster, and whether a CTA takes both KV heads of a row or one.
struct ClusterForm {
  bool both;
  int ctas, walkers;  // walkers: warps of a CTA that share a KV head's blocks

  long long total(int batch) const { return (long long)ctas * batch * (both ? 1 : kHkv); }
  int per_walker(int blocks) const { return (blocks + ctas * walkers - 1) / (ctas * walkers); }
};
// `room` SMs with `per_sm` hundredths of a CTA each; `blocks` bounds a row's blocks, lengths are on the device.
static ClusterForm cluster_form(int batch, int blocks, int sms, int room, int per_sm) {
  // Both KV heads in one CTA once three CTAs per row and head do not fit (68 rows): the two halves of a block's rows are then
  // read at about the same time (128 rows of 64 - 512 keys: 21.1 us with 3 CTAs per row, 22.5 with 2 per head).  Below that the
  // finer split per head is as fast or faster.
  const bool both = 100LL * 3 * kHkv * batch > (long long)kCmPerSm * sms;
  if (!both) return {false, cluster_size(2LL * batch, blocks, room, kCmWarps, per_sm, 8, kClMaxCluster), kCmWarps};
  // On the SMs that another kernel leaves, the places are few and eight CTAs per row fill them evenly (96 rows of up to 2048 keys
  // beside three chunks of 300, 88 SMs, six layers: 380 us, with four, which fill them 1.5 times, 396).
  if (room < sms) return {true, cluster_size(batch, blocks, room, kCmWarps / 2, per_sm, 8, 8), kCmWarps / 2};
  ClusterForm f{true, cluster_size(batch, blocks, room, kCmWarps / 2, per_sm, 4, 8), kCmWarps / 2};
  // More than four CTAs per row only beyond 24 blocks per walker, and then six where they fill the places (three to an SM) more
  // than 2.5 times, eight where they do not: a CTA that finds no block costs its start all the same.  256 rows under a table of
  // 128 blocks, filled to 1/4 - 1 and to 1/32 - 1/8 of it: 112 and 42 us with eight, 114 and 28 with four (streaming kernel 113
  // and 30); 263 blocks: 209 and 52 with eight, 212 and 44 with six (217 and 42).
  if (f.per_walker(blocks) > 24 && f.ctas < 6) f.ctas = 2LL * 6 * batch > 15LL * sms ? 6 : 8;
  return f;
}

// Whether this kernel, launched as cluster_form() says, beats the streaming kernel (paged_decode_stream.cu) on a bf16 batch.
// While CTAs have an SM each: the streaming kernel costs ~11 us whatever the batch plus its bytes at the HBM rate, this one
// ~4.5 us plus ~1.1 us per block of the longest warp.  Beyond that, where the streaming kernel's equal shares win once a CTA's
// own work gets long, by the blocks of a walker, and with an eye on rows much shorter than the table (a server that pads its
// tables), for which a CTA without a block is pure cost.  Measured at 2 - 512 rows and 24 - 512 blocks, rows of 1/4 - 1
// and of 1/32 - 1/8 of the table (us, clusters : streaming):
//   eight CTAs and more per row and head that all find a place, 16 blocks per walker: 16 rows under 512 blocks 33.3 : 35.2 and
//   10.0 : 13.4, 24 under 512 45.8 : 47.7 and 11.2 : 14.4; that do not, 32 under 400 47.8 : 48.1 and 15.7 : 14.6;
//   eight CTAs per row and head that fill the places more than twice: 67 rows under 320 71.0 : 73.4 and 22.2 : 19.0;
//   160 rows under 200, eight per row: 103.9 : 105.4 and 31.5 : 23.1; under 160, four per row, which fill the places between once
//   and 5/3 times with 20 blocks per walker: 87.6 : 89.3 and 21.5 : 21.3; with 16, under 128, 71.4 : 72.2 and 19.2 : 20.0;
//   256 rows under 256 200.0 : 204.5 and 41.0 : 35.2, under 128 106.4 : 108.2 and 27.4 : 24.5.
bool decode_cluster_pays(int batch, int table_width) {
  const int sms = decode_wide_num_ctas();
  if (sms <= 0 || batch > kClMaxRows) return false;
  const ClusterForm f = cluster_form(batch, table_width, sms, sms, kCmPerSm);
  const long long total = f.total(batch);
  const int per_walker = f.per_walker(table_width);
  if (total < sms) return 1.25 * per_walker <= 9.5 + 0.0026 * batch * table_width;  // 32 KiB per block, half of the widest on average, 6.3 TB/s
  if (f.ctas == 8 && total > 6LL * sms) return false;
  if (!f.both) return per_walker <= (f.ctas >= 8 && 100 * total <= (long long)kCmPerSm * sms ? 16 : 12);
  if (total > 3LL * sms && total < 5LL * sms) return per_walker <= 16;
  return per_walker <= (f.ctas == 6 ? 32 : 24);
}

// For the token pick a row's CTAs are one cluster, over both heads: 9 - 16 CTAs per head do not fit one, and more than ten in all
// (placed by the GPC, three or four to one) only pay while they leave places free.  Eight steps of a graph, picked here : behind: 20
// rows of 375 - 1500 keys (16 CTAs) 122 : 134 us, 25 rows 170 : 164, 28 (14) 180 : 150, 32 (12) 168 : 153, 37 of 1450 - 2900 (10)
// 303 : 313, 54 of 117 - 468 (6) 117 : 137, 8 of 50 - 200 79 : 95, 256 of 1024 - 4096 (4, both heads each) 1640 : 1662.
bool decode_cluster_picks(const DecodeParams& p) {
  const int sms = decode_wide_num_ctas();
  if (sms <= 0 || !p.pre_append || p.kv_dtype != NVJ_BF16 || p.q_dtype != NVJ_BF16 || p.kv_indptr || p.packed_rows) return false;
  const ClusterForm f = cluster_form(p.batch, p.table_width, sms, sms, kCmPerSm);
  const int members = kHkv * f.ctas;
  return f.both || members <= 10 || (members <= kClMaxCluster && 100LL * members * p.batch <= 225LL * sms);
}

int launch_decode_cluster(const DecodeParams& call, cudaStream_t stream) {
  if (call.batch > kClMaxRows) return NVJ_ERR_UNSUPPORTED;
  const int sms = decode_wide_num_ctas();
  if (sms <= 0) return NVJ_ERR_LAUNCH;
  DecodeParams p = call;
  p.early_ctas = p.new_k || p.kv_indptr || p.packed_rows || p.beside ? 0 : 3 * sms;  // three CTAs to an SM
  // (with a page list per row its width is not known here: as many CTAs as an ordinary row has use for)
  const int blocks = p.kv_indptr ? 64 : p.table_width;
  // Beside another kernel: the SMs that it leaves (cta_limit), three CTAs to each; the ones too many start when it ends (six
  // layers of 64 decode rows and two 256-token chunks, which take 32 SMs, 268 -> 259 us; 48 rows and three of 384 273 -> 255).
  // Not the few rows that get eight CTAs and more: they leave SMs free.
  ClusterForm form = cluster_form(p.batch, blocks, sms, sms, kCmPerSm);
  if (p.beside && p.cta_limit > 0 && (form.both || form.ctas < 8)) form = cluster_form(p.batch, blocks, sms, p.cta_limit, 300);
  // The CUDA-core form: eight warps, a quarter block each, two CTAs per SM (1.8: clusters do not find every SM).  More than four
  // CTAs per row and head by the table's width alone only where eight fill the places at most twice (37 rows): f32, 32 rows of
  // 2000 - 8000 keys 111 us with eight and 116 with four, of 256 - 1024 under a table of 8192 23.9 and 21.2; 128 rows of 512 - 2048
  // 115 and 109, of 256 - 1024 under 8192 77 and 63; 256 rows of 512 - 2048 223 and 203.
  const int wide = cluster_size(2LL * p.batch, blocks, sms, kClWarps * kClUnit / kBlk, 180, 16LL * p.batch <= 4LL * sms ? 8 : 4, 8);
  static PerDeviceFlags flags[8];
  const int smem = (int)sizeof(CmSmem);
  auto both = [&](auto* kernel, PerDeviceFlags& f) { return launch_clusters(kernel, f, p, dim3(form.ctas), 1, kCmThreads, smem, stream, p); };
  auto each = [&](auto* kernel, PerDeviceFlags& f, int heads_per_cluster) {
    return launch_clusters(kernel, f, p, dim3(form.ctas, heads_per_cluster), kHkv, kCmThreads, smem, stream, p);
  };
  if (p.kv_dtype == NVJ_BF16 && p.q_dtype == NVJ_BF16) {
    if (p.pick_tokens)
      return form.both ? both(decode_cluster_mma_kernel<__nv_bfloat16, true, true>, flags[6])
                       : each(decode_cluster_mma_kernel<__nv_bfloat16, false, true>, flags[7], kHkv);
    return form.both ? both(decode_cluster_mma_kernel<__nv_bfloat16, true, false>, flags[0])
                     : each(decode_cluster_mma_kernel<__nv_bfloat16, false, false>, flags[1], 1);
  }
  if (p.kv_dtype == NVJ_F16 && p.q_dtype == NVJ_F16)
    return form.both ? both(decode_cluster_mma_kernel<__half, true, false>, flags[2]) : each(decode_cluster_mma_kernel<__half, false, false>, flags[3], 1);
  if (p.kv_dtype == NVJ_F32)
    return launch_clusters(decode_cluster_kernel<float>, flags[4], p, dim3(wide), kHkv, kClThreads, cluster_smem_bytes<float>(), stream, p);
  if (p.kv_dtype == NVJ_F16)
    return launch_clusters(decode_cluster_kernel<__half>, flags[5], p, dim3(wide), kHkv, kClThreads, cluster_smem_bytes<__half>(), stream, p);
  return NVJ_ERR_UNSUPPORTED;  // bf16 cache with another query dtype: the streaming kernel on the CUDA cores
}

}  // namespace nvj
