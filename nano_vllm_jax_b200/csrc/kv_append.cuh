// Slot resolution shared by the append kernels: where token i of a batch lands in one layer of
// the paged cache, under the reference's valid-token rules (nanovllm_jax/kv_cache.py:476-564,
// nanovllm_jax/backends.py:1050-1057) and its page-table form
// (nanovllm_jax/kernels/csrc/fp32_kv_append.cu:801-841).

#pragma once

#include "nvj_common.cuh"

namespace nvj {

struct AppendParams {
  const void* new_k;
  const void* new_v;
  void* k_cache;
  void* v_cache;
  const int32_t* slot_mapping;  // slot mode
  const int32_t* valid_mask;
  const int32_t* query_start_loc;
  // page-table mode
  const int32_t* batch_indices;
  const int32_t* positions;
  const int32_t* kv_indices;
  const int32_t* kv_indptr;   // null: row b's table starts at b * table_width
  const int32_t* seq_lens;    // page-table mode, optional: rows with seq_lens[b] <= 0 are skipped
  // mapped mode (block_tables set): the slot is made here from the token's position and its row's block table
  const int32_t* block_tables;
  const int32_t* token_row_ids;  // null: rectangular batch, row = i / n_cols
  int table_rows;
  int32_t* status;
  long long num_slots;
  long long kv_indices_len;
  int n_tokens;
  int n_cols;
  int qsl_rows;
  int packed;
  int batch;
  int page_size;
  int table_width;
  int row_elems;  // num_kv_heads * head_dim
  int src_dtype;
  int dst_dtype;
};

// Flat slot of position `pos` of row `row`: floor division and a non-negative remainder, as jnp's // and % give for a
// negative position (nanovllm_jax/kv_cache.py:432-435; C's / and % would round toward zero); a negative block index
// wraps around once as NumPy / jnp indexing does, then the gather clamps.
__device__ __forceinline__ int mapped_slot(const int32_t* block_tables, int row, int pos, int table_rows, int table_width,
                                           int block_size) {
  row = row < 0 ? 0 : (row >= table_rows ? table_rows - 1 : row);
  int col = pos / block_size, off = pos % block_size;
  if (off < 0) { off += block_size; --col; }
  if (col < 0) col += table_width;
  col = col < 0 ? 0 : (col >= table_width ? table_width - 1 : col);
  return block_tables[(long long)row * table_width + col] * block_size + off;
}

// Returns the flat destination slot of token i, or -1 when the token is masked
// out or its slot lies outside the pool (the latter is flagged).
__device__ __forceinline__ long long resolve_slot(const AppendParams& p, int i) {
  long long slot;
  if (p.slot_mapping || p.block_tables) {
    // What decides about the token and what makes its slot are asked for together: one trip to memory for a mapping, two for a table
    // (three and four one after the other, most of what a small batch's append takes).
    const int mask = p.valid_mask ? p.valid_mask[i] : 1;
    const int r = p.packed ? 0 : i / p.n_cols;
    int count = 0x7fffffff, at = i;  // the token counts if at < count
    if (p.query_start_loc) {
      if (p.packed) {
        count = p.query_start_loc[p.qsl_rows];
      } else {
        if (r >= p.qsl_rows) return -1;
        count = p.query_start_loc[r + 1] - p.query_start_loc[r];
        at = i - r * p.n_cols;
      }
    }
    slot = p.slot_mapping ? p.slot_mapping[i]
                          : mapped_slot(p.block_tables, p.token_row_ids ? p.token_row_ids[i] : i / p.n_cols, p.positions[i],
                                        p.table_rows, p.table_width, p.page_size);
    if (mask == 0 || at >= count) return -1;
  } else {
    if (p.valid_mask && p.valid_mask[i] == 0) return -1;
    const int b = p.batch_indices ? p.batch_indices[i] : i;
    const int pos = p.positions[i];
    if (b < 0 || b >= p.batch || pos < 0) {
      if (p.status) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
      return -1;
    }
    if (p.seq_lens && p.seq_lens[b] <= 0) return -1;
    // the page index is bounded by the row's own page list, so a position past it cannot reach the next row's pages
    const int page = pos / p.page_size;
    const long long first = p.kv_indptr ? (long long)p.kv_indptr[b] : (long long)b * p.table_width;
    const long long pages = p.kv_indptr ? (long long)p.kv_indptr[b + 1] - first : (long long)p.table_width;
    const long long e = first + page;
    if (page >= pages || e < 0 || e >= p.kv_indices_len) {
      if (p.status) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
      return -1;
    }
    slot = (long long)p.kv_indices[e] * p.page_size + pos % p.page_size;
  }
  if (slot < 0 || slot >= p.num_slots) {
    if (p.status) atomicOr(p.status, NVJ_DEV_BAD_BLOCK_ID);
    return -1;
  }
  return slot;
}

}  // namespace nvj
