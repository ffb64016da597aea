"""Scheduler -> executor batch contract and its builders.

`ScheduledBatch` carries the fields of the reference's dataclass that this path
reads (nanovllm_jax/engine/scheduled_batch.py:11-49).  The three builders restate
the layouts `Scheduler.build_scheduled_batch`, `_build_packed_prefill_batch` and
`build_mixed_prefill_decode_batch` produce (nanovllm_jax/engine/scheduler.py:
734-1098): decode rows carry `tokens=[last]`, `positions=[num_tokens-1]`,
`seq_lens=num_tokens`; packed batches hold every query token in one row of
`token_bucket` entries with `token_row_ids`, padded with (token 0, position 0,
row 0); padded rows have an all-zero table, `seq_len 0` and `seq_id -1`.
Host lists are written into one pinned staging buffer by the host extension and moved to the device in one copy (one
pinned array and one copy per field took 0.4 ms for a 34-row mixed batch).
"""

from __future__ import annotations

from dataclasses import dataclass
from itertools import accumulate
from typing import List, Optional, Sequence as Seq

import torch

from . import host_functions

_pack_batch = host_functions.load().pack_batch


@dataclass
class ScheduledBatch:
    tokens: torch.Tensor
    positions: torch.Tensor
    seq_ids: torch.Tensor
    query_start_loc: torch.Tensor
    is_prefill: bool
    num_prefill_tokens: int
    num_decode_tokens: int
    block_tables: torch.Tensor
    seq_lens: torch.Tensor
    prefill_is_final: Optional[List[bool]] = None
    seq_ids_host: Optional[tuple] = None
    query_lens_host: Optional[tuple] = None
    seq_lens_host: Optional[tuple] = None
    block_tables_host: Optional[tuple] = None
    packed_prefill: bool = False
    token_row_ids: Optional[torch.Tensor] = None
    mixed_prefill_decode: bool = False

    @property
    def batch_size(self) -> int:
        return int(self.block_tables.shape[0] if self.packed_prefill else self.tokens.shape[0])

    @property
    def query_lens(self) -> torch.Tensor:
        return torch.diff(self.query_start_loc).to(torch.int32)


def _to_device(parts, tables, width, device):
    """The batch's int32 arrays on the device, from one staging buffer and one copy: `parts` is a list of (list of ints,
    shape), `tables` the rows' block tables (padding rows empty lists).  Returns (tensors of the parts, the [rows, width]
    table, the table as a tuple of tuples)."""
    device = torch.device(device)
    index = -1
    if device.type == "cuda":
        torch.cuda.init()
        index = torch.cuda.current_device() if device.index is None else device.index
    return _pack_batch(parts, tables, width, index)


def _tables(seqs, width: Optional[int]):
    """The rows' block tables, and the width of the batch's table: the given one or that of the longest."""
    tables = [s.block_table for s in seqs]
    return tables, width or max(1, max(map(len, tables)))


def build_decode_batch(seqs, *, max_blocks_per_seq: Optional[int] = None,
                       batch_size_bucket: Optional[int] = None, device="cuda") -> ScheduledBatch:
    """Width-1 decode batch (scheduler.py:790-803, 850-870)."""
    n = len(seqs)
    bucket = n if batch_size_bucket is None else batch_size_bucket
    if n > bucket:
        raise ValueError(f"scheduled batch has {n} seqs but bucket has {bucket}")
    tables, width = _tables(seqs, max_blocks_per_seq)
    pad = bucket - n
    zeros = [0] * pad
    lens = [s.num_tokens for s in seqs] + zeros
    seq_ids = [s.seq_id for s in seqs] + [-1] * pad
    (tokens, positions, seq_lens, qsl, ids), tab, host_tables = _to_device(
        [([s.last_token for s in seqs] + zeros, (bucket, 1)), ([s.num_tokens - 1 for s in seqs] + zeros, (bucket, 1)),
         (lens, (bucket,)), (list(range(n + 1)) + [n] * pad, (bucket + 1,)), (seq_ids, (bucket,))],
        tables + [[]] * pad, width, device)
    return ScheduledBatch(
        tokens=tokens, positions=positions, seq_ids=ids, query_start_loc=qsl, is_prefill=False, num_prefill_tokens=0,
        num_decode_tokens=n, block_tables=tab, seq_lens=seq_lens, seq_ids_host=tuple(seq_ids),
        query_lens_host=tuple([1] * n + zeros), seq_lens_host=tuple(lens), block_tables_host=host_tables)


def _pack(toks, pos, qlens, seqs, lens, finals, *, max_blocks, bucket_rows, token_bucket, device, mixed=False) -> ScheduledBatch:
    """A packed batch from its rows' tokens and positions, laid end to end (row r has qlens[r] of them)."""
    actual = len(toks)
    if actual <= 0:
        raise ValueError("packed prefill requires at least one executable token")
    token_bucket = actual if token_bucket is None else token_bucket
    if actual > token_bucket:
        raise ValueError(f"scheduled prefill needs {actual} tokens but bucket has {token_bucket}")
    pad_rows = bucket_rows - len(seqs)
    if pad_rows < 0:
        raise ValueError(f"scheduled batch has {len(seqs)} seqs but bucket has {bucket_rows}")
    tables, width = _tables(seqs, max_blocks)
    rid = []
    for r, n in enumerate(qlens):
        if n == 1:
            rid.append(r)
        else:
            rid.extend([r] * n)
    qsl = [0, *accumulate(qlens)]
    qsl.extend([actual] * pad_rows)
    lens = lens + [0] * pad_rows
    seq_ids = [s.seq_id for s in seqs] + [-1] * pad_rows
    row = (1, token_bucket)  # (the staging buffer starts as zeros: token 0, position 0, row 0 behind the last real token)
    (tokens, positions, ids, qsl_dev, lens_dev, rids), tab, host_tables = _to_device(
        [(toks, row), (pos, row), (seq_ids, (bucket_rows,)), (qsl, (bucket_rows + 1,)), (lens, (bucket_rows,)), (rid, row)],
        tables + [[]] * pad_rows, width, device)
    return ScheduledBatch(
        tokens=tokens, positions=positions, seq_ids=ids, query_start_loc=qsl_dev, is_prefill=True, num_prefill_tokens=actual,
        num_decode_tokens=0, block_tables=tab, seq_lens=lens_dev, prefill_is_final=list(finals), seq_ids_host=tuple(seq_ids),
        query_lens_host=tuple(qlens + [0] * pad_rows), seq_lens_host=tuple(lens), block_tables_host=host_tables,
        packed_prefill=True, token_row_ids=rids, mixed_prefill_decode=mixed)


def _add_row(toks, pos, qlens, lens, finals, s, start, end) -> None:
    tokens = s.token_ids[start:end]
    toks.extend(tokens)
    pos.extend(range(start, start + len(tokens)))
    qlens.append(len(tokens))
    lens.append(end)
    finals.append(end >= s.num_tokens)


def build_packed_prefill_batch(seqs, prefill_chunk_lens: Optional[Seq[int]] = None, *,
                               max_blocks_per_seq: Optional[int] = None, batch_size_bucket: Optional[int] = None,
                               token_bucket: Optional[int] = None, device="cuda") -> ScheduledBatch:
    """Packed prefill: each row runs tokens [num_cached_tokens, +chunk) (scheduler.py:774-789, 1034-1098)."""
    toks, pos, qlens, lens, finals = [], [], [], [], []
    for i, s in enumerate(seqs):
        start = s.num_cached_tokens
        chunk = s.num_tokens - start if prefill_chunk_lens is None else int(prefill_chunk_lens[i])
        if chunk <= 0:
            raise ValueError(f"Scheduled sequence {s.seq_id} has no executable tokens")
        _add_row(toks, pos, qlens, lens, finals, s, start, start + chunk)
    return _pack(toks, pos, qlens, seqs, lens, finals, max_blocks=max_blocks_per_seq,
                 bucket_rows=len(seqs) if batch_size_bucket is None else batch_size_bucket,
                 token_bucket=token_bucket, device=device)


def build_mixed_prefill_decode_batch(*, decode_seqs, prefill_seqs, prefill_chunk_lens,
                                     max_blocks_per_seq: Optional[int] = None,
                                     batch_size_bucket: Optional[int] = None,
                                     token_bucket: Optional[int] = None, device="cuda") -> ScheduledBatch:
    """Decode rows (one token each) first, then prefill chunks, in the packed form (scheduler.py:956-1032)."""
    if not decode_seqs:
        raise ValueError("mixed prefill/decode batch requires at least one decode row")
    if not prefill_seqs:
        raise ValueError("mixed prefill/decode batch requires at least one prefill row")
    if len(prefill_seqs) != len(prefill_chunk_lens):
        raise ValueError("prefill_chunk_lens length must match prefill_seqs")
    toks = [s.last_token for s in decode_seqs]
    lens = [s.num_tokens for s in decode_seqs]
    pos = [n - 1 for n in lens]
    qlens, finals = [1] * len(lens), [True] * len(lens)
    for s, c in zip(prefill_seqs, prefill_chunk_lens):
        start = s.num_cached_tokens
        chunk = min(int(c), s.num_prompt_tokens - start)
        if chunk <= 0:
            raise ValueError(f"Scheduled sequence {s.seq_id} has no executable prefill tokens")
        _add_row(toks, pos, qlens, lens, finals, s, start, start + chunk)
    seqs = list(decode_seqs) + list(prefill_seqs)
    return _pack(toks, pos, qlens, seqs, lens, finals, max_blocks=max_blocks_per_seq,
                 bucket_rows=len(seqs) if batch_size_bucket is None else batch_size_bucket,
                 token_bucket=token_bucket, device=device, mixed=True)
