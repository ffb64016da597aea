// Index-list copies on the path: whole cache blocks (prefix reuse by copy) and
// GDN hybrid-state rows (snapshot into / restore from a pool keyed by prefix
// hash), plus the per-row argmax that stands in for the sampler.
//
// The copies are HBM-bound; the algorithmic traffic is one write per pair and one
// read per distinct source.  Cache blocks move by 16-byte vector accesses, four
// independent loads in flight per thread, on a grid of (chunk group, pair, plane);
// state rows by the bulk-copy engine where they are whole 16-byte pieces.

#include "nvj_common.cuh"
#include "row_argmax.cuh"

namespace nvj {

constexpr int kCopyThreads = 256;
constexpr int kCopyUnroll = 4;
constexpr long long kCopyTileBytes = (long long)kCopyThreads * kCopyUnroll * 16;  // 16 KiB

__device__ __forceinline__ void st_cs_u4(void* p, uint4 v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}

// Copies `bytes` (multiple of 16, both pointers 16-byte aligned) with CTA `block` of `nblocks`
// moving the 16 KiB tiles block, block + nblocks, ...
__device__ __forceinline__ void copy_span16(const char* src, char* dst, long long bytes, int block, int nblocks) {
  const long long chunks = bytes >> 4;
  for (long long base = (long long)block * kCopyThreads * kCopyUnroll; base < chunks;
       base += (long long)nblocks * kCopyThreads * kCopyUnroll) {
    uint4 v[kCopyUnroll];
#pragma unroll
    for (int u = 0; u < kCopyUnroll; ++u) {
      const long long c = base + u * kCopyThreads + threadIdx.x;
      if (c < chunks) v[u] = ld_stream_u4(src + (c << 4));
    }
#pragma unroll
    for (int u = 0; u < kCopyUnroll; ++u) {
      const long long c = base + u * kCopyThreads + threadIdx.x;
      if (c < chunks) st_cs_u4(dst + (c << 4), v[u]);
    }
  }
}

__device__ __forceinline__ void copy_span1(const char* src, char* dst, long long bytes, int block, int nblocks) {
  for (long long c = (long long)block * kCopyThreads + threadIdx.x; c < bytes; c += (long long)nblocks * kCopyThreads)
    dst[c] = src[c];
}

// The (source, destination) row indices of a copy: two device arrays, or, for a handful of pairs that the host knows
// (the usual case: one restore per prefix hit), the values themselves, carried in the kernel's parameters so that no
// host-to-device copy has to run in front of the launch.
constexpr int kInlinePairs = 24;
struct SlotLists {
  const int32_t* src;
  const int32_t* dst;
  int32_t inline_src[kInlinePairs];
  int32_t inline_dst[kInlinePairs];
  __device__ __forceinline__ long long source(int i) const { return src ? src[i] : inline_src[i]; }
  __device__ __forceinline__ long long destination(int i) const { return dst ? dst[i] : inline_dst[i]; }
};

// One table of rows that are copied by index: dst_base[dst_idx[i]] <- src_base[src_idx[i]].
struct RowTable {
  const char* src_base;
  char* dst_base;
  long long row_bytes;
  int vec16;
  int blocks;  // CTAs of grid.x that work on this table
};

// Both tables of a hybrid state (recurrent and conv) in one launch; grid.y = pair, grid.x = a.blocks + b.blocks.
__global__ void __launch_bounds__(kCopyThreads)
copy_rows_kernel(RowTable a, RowTable b, long long src_rows, long long dst_rows, const __grid_constant__ SlotLists slots,
                 int32_t* status) {
  const int i = blockIdx.y;
  const long long s = slots.source(i), d = slots.destination(i);
  if (s < 0 || s >= src_rows || d < 0 || d >= dst_rows) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && status) atomicOr(status, NVJ_DEV_BAD_BLOCK_ID);
    return;
  }
  const bool first = (int)blockIdx.x < a.blocks;
  const RowTable& t = first ? a : b;
  const int block = first ? blockIdx.x : blockIdx.x - a.blocks;
  const char* src = t.src_base + s * t.row_bytes;
  char* dst = t.dst_base + d * t.row_bytes;
  if (t.vec16) copy_span16(src, dst, t.row_bytes, block, t.blocks);
  else copy_span1(src, dst, t.row_bytes, block, t.blocks);
}

// The same row copy for rows whose size is a multiple of 16 bytes, moved by the bulk-copy engine: one warp per
// CTA, a ring of kBulkStages chunks of kBulkChunk bytes in shared memory, every chunk loaded by one
// cp.async.bulk (global -> shared, completion on an mbarrier) and written back by one cp.async.bulk
// (shared -> global, tracked by a bulk group).  A thread keeps 64 KiB in flight instead of 64 bytes, which is
// what a copy of one 19 MB state row needs to reach the memory system's bandwidth: with 16-byte vector loads
// the same copy is bound by the latency of its few loads per thread.  The chunks of all pairs and both tables
// form one sequence dealt round-robin to the CTAs, the pair running fastest: pairs that share a source row (one
// stored prefix, several requests) read a chunk of it at about the same time, once from memory.  Pair after pair, the
// row had left L2 when the next pair came to it: one 19.5 MB row into 4 slots 31.7 -> 22.5 us, into 12 79.9 -> 51.2; rows
// without a shared source take the same time either way (4: 32 us).  Placed while the kernel in front still runs, which
// takes 2 - 3 us off each of the copies that a prefix hit makes one after another; 8 stages of 8 KiB are 6 - 27% slower.
constexpr int kBulkChunk = 16 * 1024;
constexpr int kBulkStages = 4;

struct BulkSmem {
  alignas(128) unsigned char stage[kBulkStages][kBulkChunk];
  alignas(8) unsigned long long full[kBulkStages];
  char* dst[kBulkStages];        // where a stage's chunk goes, and how many bytes of it (0: a pair with a bad index)
  uint32_t bytes[kBulkStages];
  int abort_flag;
};

__device__ __forceinline__ void bulk_s2g(void* gmem_dst, uint32_t smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gmem_dst), "r"(smem_src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
template <int N>
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory"); }

// `mine` chunks through the ring.  locate(src, dst) gives the next chunk's addresses and its bytes (0: leave it out).  A stage
// takes its next chunk one step after it was written back, when that store has had a chunk's time to read it.
template <class Locate>
__device__ __forceinline__ void bulk_ring(BulkSmem& sm, long long mine, int32_t* status, Locate locate) {
  auto issue_load = [&](long long k) {
    const int s = (int)(k % kBulkStages);
    const char* src = nullptr;
    char* dst = nullptr;
    const uint32_t bytes = locate(src, dst);
    sm.dst[s] = dst;
    sm.bytes[s] = bytes;
    const uint32_t bar = smem_u32(&sm.full[s]);
    if (bytes > 0) {
      mbar_arrive_expect_tx(bar, bytes);
      bulk_g2s(smem_u32(sm.stage[s]), src, bytes, bar);
    } else {
      mbar_arrive(bar);
    }
  };
  long long issued = 0;
  for (; issued < mine && issued < kBulkStages; ++issued) issue_load(issued);
  for (long long k = 0; k < mine; ++k) {
    const int s = (int)(k % kBulkStages);
    if (!mbar_wait(smem_u32(&sm.full[s]), (uint32_t)(k / kBulkStages) & 1u, &sm.abort_flag, status)) break;
    if (sm.bytes[s] > 0) {
      fence_proxy_async_all();
      bulk_s2g(sm.dst[s], smem_u32(sm.stage[s]), sm.bytes[s]);
    }
    bulk_commit();
    if (k > 0 && issued < mine) {
      bulk_wait_read<1>();  // the store before this one has read its stage: it can take the next chunk
      issue_load(issued++);
    }
  }
  bulk_wait_all<0>();
  if (sm.abort_flag) {  // only after a timeout can loads still be in flight: hold the shared memory until they have landed
    const unsigned long long t0 = global_timer_ns();
    for (long long k = issued > kBulkStages ? issued - kBulkStages : 0; k < issued; ++k)
      while (!mbar_try_wait(smem_u32(&sm.full[k % kBulkStages]), (uint32_t)(k / kBulkStages) & 1u) &&
             global_timer_ns() - t0 < kWaitLimitNs) {
      }
  }
}

__device__ __forceinline__ BulkSmem& bulk_smem() {
  extern __shared__ unsigned char bulk_smem_raw[];
  return *reinterpret_cast<BulkSmem*>((reinterpret_cast<uintptr_t>(bulk_smem_raw) + 127) & ~(uintptr_t)127);
}
__device__ __forceinline__ void bulk_ring_init(BulkSmem& sm) {
  sm.abort_flag = 0;
  for (int s = 0; s < kBulkStages; ++s) mbar_init(smem_u32(&sm.full[s]), 1);
  mbar_fence_init();
}

__global__ void __launch_bounds__(32)
copy_rows_bulk_kernel(RowTable a, RowTable b, long long src_rows, long long dst_rows, const __grid_constant__ SlotLists slots,
                      int n_pairs, int32_t* status) {
  BulkSmem& sm = bulk_smem();
  if (threadIdx.x != 0) return;  // one thread drives the copy engine; the warp exists only to own the shared memory
  bulk_ring_init(sm);
  const long long chunks_a = (a.row_bytes + kBulkChunk - 1) / kBulkChunk, chunks_b = (b.row_bytes + kBulkChunk - 1) / kBulkChunk;
  const long long total = (chunks_a + chunks_b) * n_pairs, first = blockIdx.x, stride = gridDim.x;
  const long long mine = first < total ? (total - first + stride - 1) / stride : 0;
  long long row_chunk = first / n_pairs;
  int pair = (int)(first - row_chunk * n_pairs);
  const int chunk_step = (int)gridDim.x / n_pairs, pair_step = (int)gridDim.x - chunk_step * n_pairs;
  pdl_wait();
  pdl_release();
  bulk_ring(sm, mine, status, [&](const char*& src, char*& dst) -> uint32_t {
    const long long si = slots.source(pair), di = slots.destination(pair), chunk = row_chunk;
    row_chunk += chunk_step;
    pair += pair_step;
    if (pair >= n_pairs) {
      pair -= n_pairs;
      ++row_chunk;
    }
    if (si < 0 || si >= src_rows || di < 0 || di >= dst_rows) {
      if (status) atomicOr(status, NVJ_DEV_BAD_BLOCK_ID);
      return 0;
    }
    const bool second = chunk >= chunks_a;
    const long long row_bytes = second ? b.row_bytes : a.row_bytes, off = (second ? chunk - chunks_a : chunk) * kBulkChunk;
    src = (second ? b.src_base : a.src_base) + si * row_bytes + off;
    dst = (second ? b.dst_base : a.dst_base) + di * row_bytes + off;
    const long long left = row_bytes - off;
    return (uint32_t)(left < kBulkChunk ? left : kBulkChunk);
  });
}

// Block copy across layers and K/V: grid.y = pair, grid.z = layer * 2 + (0: K, 1: V).  (The bulk-copy ring above moves 16 KiB
// blocks no faster: 128 pairs of 6 layers 14.3 us against 12.3, 768 pairs 41 against 35.)
__global__ void __launch_bounds__(kCopyThreads)
copy_blocks_kernel(char* k_cache, char* v_cache, long long num_blocks, long long block_bytes,
                   long long layer_stride, const int32_t* src_ids, const int32_t* dst_ids, int vec16,
                   int32_t* status) {
  pdl_wait();
  pdl_release();
  const int i = blockIdx.y;
  const long long s = src_ids[i], d = dst_ids[i];
  if (s < 0 || s >= num_blocks || d < 0 || d >= num_blocks) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.z == 0 && status)
      atomicOr(status, NVJ_DEV_BAD_BLOCK_ID);
    return;
  }
  if (s == d) return;
  char* base = (blockIdx.z & 1) ? v_cache : k_cache;
  base += (long long)(blockIdx.z >> 1) * layer_stride;
  if (vec16) copy_span16(base + s * block_bytes, base + d * block_bytes, block_bytes, blockIdx.x, gridDim.x);
  else copy_span1(base + s * block_bytes, base + d * block_bytes, block_bytes, blockIdx.x, gridDim.x);
}

// One CTA per row.  With seq_lens the row's resident decode metadata is advanced in the same launch, as
// advance_decode_metadata_kernel would (the tail of a decode step whose attention ran in pre-append form).
__global__ void __launch_bounds__(kArgmaxThreads)
row_argmax_kernel(const float* x, int row_len, int32_t* tokens, int32_t* seq_lens, int32_t* positions, long long capacity,
                  int32_t* status) {
  pdl_wait();
  pdl_release();
  const int token = row_argmax_cta(x + (long long)blockIdx.x * row_len, row_len);
  if (threadIdx.x == 0) {
    tokens[blockIdx.x] = token;
    if (seq_lens) advance_row(seq_lens, positions, blockIdx.x, capacity, status);
  }
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Opt the bulk row-copy kernel into its 64 KiB of dynamic shared memory, once per device.
static bool bulk_copy_ready() {
  static PerDeviceFlags opted_in;
  return once_per_device(opted_in, [](int) {
    return cudaFuncSetAttribute(copy_rows_bulk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(BulkSmem) + 128) == cudaSuccess;
  });
}

static int sm_count() {
  static PerDeviceFlags cached;  // 0 = not queried yet
  const int dev = current_device();
  if (dev < 0) return 0;
  int n = cached.v[dev].load(std::memory_order_acquire);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
    cached.v[dev].store(n, std::memory_order_release);
  }
  return n;
}

static int grid_x_for(long long bytes, int pairs) {
  // Enough CTAs to fill the machine a few times over, never more than one per tile.
  long long tiles = (bytes + kCopyTileBytes - 1) / kCopyTileBytes;
  long long want = (148LL * 16 + pairs - 1) / pairs;
  long long gx = tiles < want ? tiles : want;
  return gx < 1 ? 1 : (int)gx;
}

static RowTable row_table(const void* src, void* dst, long long row_bytes, int pairs) {
  RowTable t{};
  if (!src || !dst || row_bytes == 0) return t;  // blocks = 0: no CTA works on it
  t.src_base = static_cast<const char*>(src);
  t.dst_base = static_cast<char*>(dst);
  t.row_bytes = row_bytes;
  t.vec16 = aligned16(src) && aligned16(dst) && row_bytes % 16 == 0;
  t.blocks = grid_x_for(row_bytes, pairs);
  return t;
}

// One decode step of the batch metadata, on the device: every active row (seq_len > 0) grows by
// the token it is about to append; its position is the old length.  Rows that would outgrow
// their block table are flagged and left alone.
__global__ void advance_decode_metadata_kernel(int32_t* seq_lens, int32_t* positions, int batch, long long capacity,
                                               int32_t* status) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  advance_row(seq_lens, positions, b, capacity, status);
}

}  // namespace nvj

extern "C" int nvj_abi_version(void) { return NVJ_ABI_VERSION; }

extern "C" const char* nvj_status_string(int status) {
  switch (status) {
    case NVJ_OK: return "ok";
    case NVJ_ERR_INVALID_ARGUMENT: return "invalid argument";
    case NVJ_ERR_UNSUPPORTED: return "unsupported shape or dtype";
    case NVJ_ERR_LAUNCH: return "kernel launch failed";
    case NVJ_ERR_WORKSPACE: return "workspace missing or too small";
    case NVJ_ERR_TOO_LARGE: return "size exceeds a built-in limit of this entry point";
    default: return "unknown status";
  }
}

extern "C" int nvj_copy_blocks(void* k_cache, void* v_cache, int num_layers, int64_t num_blocks,
                               int64_t block_bytes, int64_t layer_stride_bytes,
                               const int32_t* src_ids, const int32_t* dst_ids, int n_pairs,
                               int32_t* status, nvj_stream_t stream) {
  using namespace nvj;
  if (num_layers < 0 || num_blocks < 0 || block_bytes < 0 || n_pairs < 0 || layer_stride_bytes < 0)
    return NVJ_ERR_INVALID_ARGUMENT;
  if (n_pairs == 0 || num_layers == 0 || block_bytes == 0) return NVJ_OK;
  if (!k_cache || !v_cache || !src_ids || !dst_ids) return NVJ_ERR_INVALID_ARGUMENT;
  if (n_pairs > 65535 || num_layers * 2 > 65535) return NVJ_ERR_UNSUPPORTED;
  const int vec16 = aligned16(k_cache) && aligned16(v_cache) && block_bytes % 16 == 0 &&
                    layer_stride_bytes % 16 == 0;
  dim3 grid(grid_x_for(block_bytes, n_pairs * num_layers * 2), n_pairs, num_layers * 2);
  const cudaError_t e = launch_after(copy_blocks_kernel, grid, kCopyThreads, 0, static_cast<cudaStream_t>(stream),
                                     static_cast<char*>(k_cache), static_cast<char*>(v_cache), num_blocks, block_bytes,
                                     layer_stride_bytes, src_ids, dst_ids, vec16, status);
  return e == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

static int hybrid_copy(const void* conv_src, void* conv_dst, int64_t conv_row_bytes,
                       const void* rec_src, void* rec_dst, int64_t rec_row_bytes,
                       int64_t src_rows, int64_t dst_rows, const int32_t* src_slots,
                       const int32_t* dst_slots, int n, bool slots_on_host, int32_t* status, nvj_stream_t stream) {
  using namespace nvj;
  if (n < 0 || conv_row_bytes < 0 || rec_row_bytes < 0 || src_rows < 0 || dst_rows < 0)
    return NVJ_ERR_INVALID_ARGUMENT;
  if (n == 0) return NVJ_OK;
  if (!src_slots || !dst_slots) return NVJ_ERR_INVALID_ARGUMENT;
  if (n > 65535) return NVJ_ERR_UNSUPPORTED;
  SlotLists slots{};
  if (slots_on_host) {
    if (n > kInlinePairs) return NVJ_ERR_TOO_LARGE;
    for (int i = 0; i < n; ++i) { slots.inline_src[i] = src_slots[i]; slots.inline_dst[i] = dst_slots[i]; }
  } else {
    slots.src = src_slots;
    slots.dst = dst_slots;
  }
  if ((conv_src == nullptr) != (conv_dst == nullptr) || (rec_src == nullptr) != (rec_dst == nullptr))
    return NVJ_ERR_INVALID_ARGUMENT;
  const RowTable rec = row_table(rec_src, rec_dst, rec_row_bytes, n);
  const RowTable conv = row_table(conv_src, conv_dst, conv_row_bytes, n);
  if (rec.blocks + conv.blocks == 0) return NVJ_OK;
  // rows that the bulk-copy engine can move (16-byte aligned, sizes multiples of 16 bytes) go through it
  const bool bulk_ok = (rec.blocks == 0 || rec.vec16) && (conv.blocks == 0 || conv.vec16) && bulk_copy_ready();
  if (bulk_ok) {
    const long long chunks = ((rec.row_bytes + kBulkChunk - 1) / kBulkChunk + (conv.row_bytes + kBulkChunk - 1) / kBulkChunk) * n;
    const int sms = sm_count();
    const long long cap = (long long)(sms > 0 ? sms : 148) * 3;  // three CTAs of 64 KiB shared memory per SM
    const int ctas = (int)(chunks < cap ? chunks : cap);
    const cudaError_t e = launch_after(copy_rows_bulk_kernel, ctas, 32, sizeof(BulkSmem) + 128, static_cast<cudaStream_t>(stream), rec,
                                       conv, src_rows, dst_rows, slots, n, status);
    return e == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
  }
  dim3 grid(rec.blocks + conv.blocks, n, 1);
  copy_rows_kernel<<<grid, kCopyThreads, 0, static_cast<cudaStream_t>(stream)>>>(rec, conv, src_rows, dst_rows, slots, status);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

extern "C" int nvj_hybrid_snapshot(const void* conv_table, void* conv_pool, int64_t conv_row_bytes,
                                   const void* rec_table, void* rec_pool, int64_t rec_row_bytes,
                                   int64_t table_rows, int64_t pool_rows,
                                   const int32_t* table_slots, const int32_t* pool_slots, int n,
                                   int32_t* status, nvj_stream_t stream) {
  return hybrid_copy(conv_table, conv_pool, conv_row_bytes, rec_table, rec_pool, rec_row_bytes,
                     table_rows, pool_rows, table_slots, pool_slots, n, false, status, stream);
}

extern "C" int nvj_hybrid_snapshot_host_slots(const void* conv_table, void* conv_pool, int64_t conv_row_bytes,
                                              const void* rec_table, void* rec_pool, int64_t rec_row_bytes,
                                              int64_t table_rows, int64_t pool_rows,
                                              const int32_t* table_slots, const int32_t* pool_slots, int n,
                                              int32_t* status, nvj_stream_t stream) {
  return hybrid_copy(conv_table, conv_pool, conv_row_bytes, rec_table, rec_pool, rec_row_bytes,
                     table_rows, pool_rows, table_slots, pool_slots, n, true, status, stream);
}

extern "C" int nvj_hybrid_restore(void* conv_table, const void* conv_pool, int64_t conv_row_bytes,
                                  void* rec_table, const void* rec_pool, int64_t rec_row_bytes,
                                  int64_t table_rows, int64_t pool_rows,
                                  const int32_t* table_slots, const int32_t* pool_slots, int n,
                                  int32_t* status, nvj_stream_t stream) {
  return hybrid_copy(conv_pool, conv_table, conv_row_bytes, rec_pool, rec_table, rec_row_bytes,
                     pool_rows, table_rows, pool_slots, table_slots, n, false, status, stream);
}

extern "C" int nvj_hybrid_restore_host_slots(void* conv_table, const void* conv_pool, int64_t conv_row_bytes,
                                             void* rec_table, const void* rec_pool, int64_t rec_row_bytes,
                                             int64_t table_rows, int64_t pool_rows,
                                             const int32_t* table_slots, const int32_t* pool_slots, int n,
                                             int32_t* status, nvj_stream_t stream) {
  return hybrid_copy(conv_pool, conv_table, conv_row_bytes, rec_pool, rec_table, rec_row_bytes,
                     pool_rows, table_rows, pool_slots, table_slots, n, true, status, stream);
}

extern "C" int nvj_advance_decode_metadata(int32_t* seq_lens, int32_t* positions, int batch,
                                           int table_width, int block_size, int32_t* status,
                                           nvj_stream_t stream) {
  using namespace nvj;
  if (batch < 0 || table_width < 0 || block_size <= 0) return NVJ_ERR_INVALID_ARGUMENT;
  if (batch == 0) return NVJ_OK;
  if (!seq_lens || !positions) return NVJ_ERR_INVALID_ARGUMENT;
  advance_decode_metadata_kernel<<<(batch + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      seq_lens, positions, batch, (long long)table_width * block_size, status);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

extern "C" int nvj_copy_many_async(void* const* dst, const void* const* src, const size_t* bytes, int n,
                                   nvj_stream_t stream) {
  if (n < 0 || (n > 0 && (!dst || !src || !bytes))) return NVJ_ERR_INVALID_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  for (int i = 0; i < n; ++i) {
    if (bytes[i] == 0) continue;
    if (!dst[i] || !src[i]) return NVJ_ERR_INVALID_ARGUMENT;
    if (cudaMemcpyAsync(dst[i], src[i], bytes[i], cudaMemcpyDefault, s) != cudaSuccess) return NVJ_ERR_LAUNCH;
  }
  return NVJ_OK;
}

namespace nvj {

// A step's operands out of pinned host memory, all of them in one launch.  Bound by the PCIe round trip (~2 us) and rate: every
// thread has four 16-byte loads in flight, a CTA 16 KiB, and 28 CTAs ask for the 460 KB of a 64-row step at once.  Six copies by
// the copy engines took 42 us on two streams, most of it the engines' latency per copy; this takes ~14.  The loads are volatile:
// the host writes these buffers between the launches.
constexpr int kStageMost = 8, kStageThreads = 256, kStagePer = 4, kStageCtas = 64;
struct StageList {
  const uint4* src[kStageMost];
  uint4* dst[kStageMost];
  long long end[kStageMost];  // 16-byte pieces of the pairs up to this one
  int last_words[kStageMost];  // 4-byte words of the pair's last piece
  int n;
};
__global__ void __launch_bounds__(kStageThreads) stage_in_kernel(const __grid_constant__ StageList list) {
  const long long pieces = list.end[list.n - 1];
  constexpr long long kSpan = kStageThreads * kStagePer;
  for (long long base = blockIdx.x * kSpan + threadIdx.x; base < pieces; base += gridDim.x * kSpan) {
    uint4 x[kStagePer];
    uint4* to[kStagePer];
    int words[kStagePer];
#pragma unroll
    for (int k = 0; k < kStagePer; ++k) {
      long long i = base + (long long)k * kStageThreads;
      to[k] = nullptr;
      if (i >= pieces) continue;
      int e = 0;
      while (i >= list.end[e]) ++e;
      words[k] = i == list.end[e] - 1 ? list.last_words[e] : 4;
      if (e > 0) i -= list.end[e - 1];
      to[k] = list.dst[e] + i;
      if (words[k] == 4) {
        x[k] = __ldcv(list.src[e] + i);
      } else {
        const unsigned* s = reinterpret_cast<const unsigned*>(list.src[e] + i);
        x[k].x = __ldcv(s);
        if (words[k] > 1) x[k].y = __ldcv(s + 1);
        if (words[k] > 2) x[k].z = __ldcv(s + 2);
      }
    }
#pragma unroll
    for (int k = 0; k < kStagePer; ++k) {
      if (!to[k]) continue;
      if (words[k] == 4) {
        *to[k] = x[k];
      } else {
        unsigned* d = reinterpret_cast<unsigned*>(to[k]);
        d[0] = x[k].x;
        if (words[k] > 1) d[1] = x[k].y;
        if (words[k] > 2) d[2] = x[k].z;
      }
    }
  }
}

// The device's address of a pinned host buffer, null for anything else.  (Both ends: a buffer may be registered in part.)
static const void* pinned_device_address(const void* p, size_t bytes) {
  cudaPointerAttributes first, last;
  if (cudaPointerGetAttributes(&first, p) != cudaSuccess ||
      cudaPointerGetAttributes(&last, static_cast<const char*>(p) + bytes - 1) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  if (first.type != cudaMemoryTypeHost || last.type != cudaMemoryTypeHost || !first.devicePointer ||
      static_cast<const char*>(last.devicePointer) - static_cast<const char*>(first.devicePointer) != (ptrdiff_t)(bytes - 1))
    return nullptr;
  return first.devicePointer;
}

}  // namespace nvj

extern "C" int nvj_stage_in(void* const* dst, const void* const* src, const size_t* bytes, int n, nvj_stream_t stream) {
  using namespace nvj;
  if (n < 0 || (n > 0 && (!dst || !src || !bytes))) return NVJ_ERR_INVALID_ARGUMENT;
  if (n > kStageMost) return NVJ_ERR_UNSUPPORTED;
  StageList list{};
  long long pieces = 0;
  for (int i = 0; i < n; ++i) {
    if (bytes[i] == 0) continue;
    if (!dst[i] || !src[i]) return NVJ_ERR_INVALID_ARGUMENT;
    const void* from = (bytes[i] & 3) || !aligned16(dst[i]) ? nullptr : pinned_device_address(src[i], bytes[i]);
    if (!from || !aligned16(from)) return NVJ_ERR_UNSUPPORTED;
    list.src[list.n] = static_cast<const uint4*>(from);
    list.dst[list.n] = static_cast<uint4*>(dst[i]);
    pieces += (long long)((bytes[i] + 15) >> 4);
    list.last_words[list.n] = (bytes[i] & 15) ? (int)((bytes[i] & 15) >> 2) : 4;
    list.end[list.n++] = pieces;
  }
  if (list.n == 0) return NVJ_OK;
  const long long ctas = (pieces + kStageThreads * kStagePer - 1) / (kStageThreads * kStagePer);
  stage_in_kernel<<<(int)(ctas < kStageCtas ? ctas : kStageCtas), kStageThreads, 0, static_cast<cudaStream_t>(stream)>>>(list);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

extern "C" int nvj_row_argmax(const float* x, int rows, int row_len, int32_t* tokens,
                              nvj_stream_t stream) {
  using namespace nvj;
  if (rows < 0 || row_len <= 0) return NVJ_ERR_INVALID_ARGUMENT;
  if (rows == 0) return NVJ_OK;
  if (!x || !tokens) return NVJ_ERR_INVALID_ARGUMENT;
  launch_after(row_argmax_kernel, rows, kArgmaxThreads, 0, static_cast<cudaStream_t>(stream), x, row_len, tokens, nullptr, nullptr, 0, nullptr);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}

extern "C" int nvj_row_argmax_advance(const float* x, int rows, int row_len, int32_t* tokens, int32_t* seq_lens,
                                      int32_t* positions, int table_width, int block_size, int32_t* status,
                                      nvj_stream_t stream) {
  using namespace nvj;
  if (rows < 0 || row_len <= 0 || table_width < 0 || block_size <= 0) return NVJ_ERR_INVALID_ARGUMENT;
  if (rows == 0) return NVJ_OK;
  if (!x || !tokens || !seq_lens) return NVJ_ERR_INVALID_ARGUMENT;
  launch_after(row_argmax_kernel, rows, kArgmaxThreads, 0, static_cast<cudaStream_t>(stream), x, row_len, tokens, seq_lens, positions,
                                                                                   (long long)table_width * block_size, status);
  return cudaGetLastError() == cudaSuccess ? NVJ_OK : NVJ_ERR_LAUNCH;
}
