"""Host-side block allocator with hash-chained prefix reuse.

Behaviour and public names follow nanovllm_jax/engine/block_manager.py:12-387 so
the reference scheduler can drive it unchanged: reference-counted blocks, one
xxh64 digest per *full* block chained on the previous block's digest, a
`hash_to_block_id` map that only holds blocks whose KV rows were actually
computed (publish after compute), and look-ahead slot reservation for decode.
Prefix reuse is sharing by reference count; nothing is copied on the device.

The hash must be bit-identical to the reference's
(block_manager.py:49-56), and is computed by the host extension for a whole token list at a time
(one Python-level digest per block took 1.5 us, 16 tokens of it 0.06 us there): xxh64 over `prefix.to_bytes(8, "little")` (when a
prefix exists) followed by the token ids as native int64 bytes.
"""

from __future__ import annotations

from typing import Dict, List, Optional, Set

import numpy as np
import xxhash

from ..kv_cache import BlockTables
from . import host_functions

NO_HASH = -1
_host = host_functions.load()
_hash_chain = _host.hash_chain


class Block:
    """One physical cache block: owner count, content digest, the tokens it holds."""

    __slots__ = ("block_id", "ref_count", "hash", "token_ids")

    def __init__(self, block_id: int):
        self.block_id = block_id
        self.ref_count = 0
        self.hash = NO_HASH
        self.token_ids: List[int] = []

    def update(self, hash_val: int, token_ids: List[int]) -> None:
        self.hash = hash_val
        self.token_ids = token_ids

    def reset(self) -> None:
        self.ref_count = 1
        self.hash = NO_HASH
        self.token_ids = []


class _FreeList:
    """FIFO of free block ids with O(1) removal of an arbitrary id.

    A list and the index of its head, so that a sequence's blocks leave it as one slice and come back as one.  Removing an id
    from the middle (a cached block is taken again: rare) leaves its entry in the queue as a stale one, which the head skips
    when it gets there; an id's stale entries always lie in front of its live one.  Callers add only ids that are not free and
    remove only free ones.  An id is free exactly when it is not in `used` (the manager's set of owned blocks, which it keeps in
    step), so that asking for one costs a look-up.
    """

    def __init__(self, ids: range, used: Set[int]):
        self._queue: List[int] = list(ids)
        self._ids = ids
        self._used = used
        self._head = 0
        self._stale: Dict[int, int] = {}  # id -> entries to skip
        self._len = len(self._queue)

    def __len__(self) -> int:
        return self._len

    def __contains__(self, block_id: int) -> bool:
        return block_id in self._ids and block_id not in self._used

    def __iter__(self):
        stale = dict(self._stale)
        for block_id in self._queue[self._head:]:
            if stale.get(block_id, 0) > 0:
                stale[block_id] -= 1
            else:
                yield block_id

    def _advance(self, n: int) -> None:
        self._head += n
        if self._head > 256 and 2 * self._head > len(self._queue):
            del self._queue[:self._head]
            self._head = 0

    def _skip_stale(self) -> None:
        stale = self._stale
        while stale and self._head < len(self._queue):
            block_id = self._queue[self._head]
            n = stale.get(block_id, 0)
            if n == 0:
                return
            if n == 1:
                del stale[block_id]
            else:
                stale[block_id] = n - 1
            self._advance(1)

    def __getitem__(self, index: int) -> int:
        if index != 0:
            raise IndexError("only the head of the free list is addressable")
        if not self._len:
            raise StopIteration("no free block left")
        self._skip_stale()
        return self._queue[self._head]

    def remove(self, block_id: int) -> None:
        self._len -= 1
        self._stale[block_id] = self._stale.get(block_id, 0) + 1

    def append(self, block_id: int) -> None:
        self._queue.append(block_id)
        self._len += 1

    def extend(self, block_ids: List[int]) -> None:
        self._queue.extend(block_ids)
        self._len += len(block_ids)

    def take(self, n: int) -> List[int]:
        """Remove and return the first n ids; StopIteration, and nothing removed, when there are fewer."""
        if n > self._len:
            raise StopIteration("no free block left")
        out: List[int] = []
        while self._stale and len(out) < n:
            self._skip_stale()
            out.append(self._queue[self._head])
            self._advance(1)
        rest = n - len(out)
        out += self._queue[self._head:self._head + rest]
        self._advance(rest)
        self._len -= n
        return out


class BlockManager:
    def __init__(self, num_blocks: int, block_size: int):
        self.block_size = block_size
        self.blocks: List[Block] = [Block(i) for i in range(num_blocks)]
        self.hash_to_block_id: Dict[int, int] = {}
        self.used_block_ids: Set[int] = set()
        self.free_block_ids = _FreeList(range(num_blocks), self.used_block_ids)

    # ------------------------------------------------------------------ hashing
    @classmethod
    def compute_hash(cls, token_ids: List[int], prefix: int = NO_HASH) -> int:
        one = _hash_chain(token_ids, len(token_ids), 1, prefix) if token_ids else None
        if one is not None:
            return one[0]
        h = xxhash.xxh64()
        if prefix != NO_HASH:
            h.update(int(prefix).to_bytes(8, "little"))
        h.update(np.asarray(token_ids, dtype=np.int64).tobytes())
        return h.intdigest()

    def _digests(self, seq) -> List[int]:
        """Chained digests of the sequence's full blocks."""
        bs = self.block_size
        full = min(seq.num_tokens, len(seq.token_ids)) // bs
        chain = _hash_chain(seq.token_ids, bs, full, NO_HASH)
        if chain is None:  # not a plain list of integers
            chain, h = [], NO_HASH
            for idx in range(full):
                h = self.compute_hash(seq.token_ids[idx * bs:(idx + 1) * bs], h)
                chain.append(h)
        return chain

    def _num_blocks(self, seq) -> int:
        return -(-seq.num_tokens // self.block_size)

    def _lookup(self, h: int, token_ids: List[int]) -> int:
        """Published block holding exactly these tokens under this digest, else -1."""
        bid = self.hash_to_block_id.get(h, -1)
        if bid == -1:
            return -1
        blk = self.blocks[bid]
        return bid if (blk.hash == h and blk.token_ids == token_ids) else -1

    # ------------------------------------------------------------------ block state changes
    def _take_fresh(self, block_id: int) -> Block:
        blk = self.blocks[block_id]
        assert blk.ref_count == 0
        if blk.hash != NO_HASH and self.hash_to_block_id.get(blk.hash) == block_id:
            del self.hash_to_block_id[blk.hash]  # its old content is about to be overwritten
        blk.reset()
        self.free_block_ids.remove(block_id)
        self.used_block_ids.add(block_id)
        return blk

    def _take_cached(self, block_id: int) -> Block:
        blk = self.blocks[block_id]
        assert blk.ref_count == 0
        blk.ref_count = 1  # content and digest stay: the rows are still valid
        self.free_block_ids.remove(block_id)
        self.used_block_ids.add(block_id)
        return blk

    def _release(self, block_id: int) -> None:
        assert self.blocks[block_id].ref_count == 0
        self.used_block_ids.remove(block_id)
        self.free_block_ids.append(block_id)

    # aliases under the reference's private names, which its tests reach for
    _allocate_block = _take_fresh
    _reuse_cached_block = _take_cached
    _deallocate_block = _release
    _cached_block_id = _lookup

    # ------------------------------------------------------------------ prefix queries
    def cached_prefix_info(self, seq, *, cacheable_hashes: Optional[Set[int]] = None):
        """(reusable tokens, digest of that prefix): longest run of published full blocks.

        With `cacheable_hashes` the run is cut back to the longest prefix whose own
        chained digest is in the set (hybrid models need the GDN state of exactly
        that prefix).
        """
        hits, best_hash, _ = self._cached_run(seq, cacheable_hashes)
        return len(hits) * self.block_size, best_hash

    def _cached_run(self, seq, cacheable_hashes, digests=None):
        """(ids of the published blocks of the longest reusable prefix, its digest, how many of them a live sequence holds).
        Without `digests` the walk takes them as far as it goes, which is one block beyond the published ones."""
        tokens = seq.token_ids if type(seq.token_ids) is list else list(seq.token_ids)
        full = min(seq.num_tokens, len(tokens)) // self.block_size
        run = _host.cached_run(tokens, digests, self.block_size, full, self.hash_to_block_id, self.blocks, cacheable_hashes,
                               self.used_block_ids)
        return self._cached_run(seq, cacheable_hashes, self._digests(seq)) if run is None else run

    def _num_required_blocks(self, seq, *, use_prefix_cache=True, cacheable_hashes=None) -> int:
        need = self._num_blocks(seq)
        if use_prefix_cache:
            need -= self._cached_run(seq, cacheable_hashes)[2]  # shared with a live sequence: costs no free block
        return need

    def can_allocate(self, seq, *, use_prefix_cache=True, cacheable_hashes=None) -> bool:
        return len(self.free_block_ids) >= self._num_required_blocks(
            seq, use_prefix_cache=use_prefix_cache, cacheable_hashes=cacheable_hashes)

    # ------------------------------------------------------------------ allocate / free
    def allocate(self, seq, *, use_prefix_cache=True, cacheable_hashes=None) -> None:
        assert not seq.block_table
        seq.block_size = self.block_size
        seq.num_cached_tokens = 0
        seq.cached_prefix_hash = None
        seq.cached_prefix_hybrid_seeded = False
        seq.prefix_cache_enabled = bool(use_prefix_cache)
        tokens = seq.token_ids
        done = _host.allocate(seq, tokens, self.block_size, min(seq.num_tokens, len(tokens)) // self.block_size, self._num_blocks(seq),
                              self.hash_to_block_id, self.blocks, cacheable_hashes, self.used_block_ids, use_prefix_cache,
                              seq.block_table, self.free_block_ids.take, self._take_cached, NO_HASH)
        if done is not None:
            seq.cached_prefix_hash = done[0] if seq.num_cached_tokens > 0 else None
            return
        digests = self._digests(seq)
        hits, cached_hash, _ = self._cached_run(seq, cacheable_hashes, digests) if use_prefix_cache else ([], None, 0)
        blocks, used, free, bs, tokens, table = (self.blocks, self.used_block_ids, self.free_block_ids, self.block_size,
                                                 seq.token_ids, seq.block_table)
        for bid in _host.add_owner(blocks, hits, used):
            self._take_cached(bid)
        table.extend(hits)
        seq.num_cached_tokens = len(hits) * bs
        first = len(hits)
        fresh = free.take(self._num_blocks(seq) - first)
        _host.take_fresh(blocks, fresh, first, digests, tokens if type(tokens) is list else list(tokens), bs, self.hash_to_block_id,
                         NO_HASH)
        used.update(fresh)
        table.extend(fresh)
        seq.cached_prefix_hash = cached_hash if seq.num_cached_tokens > 0 else None

    def deallocate(self, seq) -> None:
        gone = _host.drop_owner(self.blocks, seq.block_table)
        self.used_block_ids.difference_update(gone)
        self.free_block_ids.extend(gone)
        seq.num_cached_tokens = 0
        seq.cached_prefix_hash = None
        seq.cached_prefix_hybrid_seeded = False
        seq.prefix_cache_enabled = False
        seq.block_table.clear()

    # ------------------------------------------------------------------ decode growth
    def _blocks_for(self, tokens: int) -> int:
        return -(-tokens // self.block_size)

    def can_append(self, seq) -> bool:
        return self.can_append_slots(seq, 1)

    def can_append_slots(self, seq, num_slots: int) -> bool:
        target = len(seq) + max(0, int(num_slots) - 1)
        return len(self.free_block_ids) >= max(0, self._blocks_for(target) - len(seq.block_table))

    def may_append(self, seq) -> None:
        self.may_append_slots(seq, 1)

    def may_append_slots(self, seq, num_slots: int) -> None:
        table, n, bs = seq.block_table, len(seq), self.block_size
        if n % bs and (n + max(0, int(num_slots) - 1) + bs - 1) // bs <= len(table):
            return  # no block is complete and the table has room: nearly every row of nearly every step
        if self._blocks_for(len(seq)) > len(table):
            last = len(table) - 1
            self._record_completed_block_hash(seq, last)
            if self.blocks[table[-1]].hash == NO_HASH and not seq.block_has_unmaterialized_device_tokens(last):
                raise AssertionError("completed block hash was not recorded")
            table.append(self._take_fresh(self.free_block_ids[0]).block_id)
        if len(seq) % self.block_size == 0:
            self._record_completed_block_hash(seq, len(seq) // self.block_size - 1)
        want = self._blocks_for(len(seq) + max(0, int(num_slots) - 1))
        while len(table) < want:
            table.append(self._take_fresh(self.free_block_ids[0]).block_id)

    def trim_append_slots(self, seq, num_slots: int) -> None:
        table = seq.block_table
        want = self._blocks_for(len(seq) + max(0, int(num_slots) - 1))
        while len(table) > want:
            blk = self.blocks[table.pop()]
            if blk.hash != NO_HASH or blk.token_ids:
                raise AssertionError("cannot trim a materialized KV block")
            blk.ref_count -= 1
            self._release(blk.block_id)

    def commit_processed_token(self, seq) -> None:
        if len(seq) % self.block_size == 0:
            self._record_completed_block_hash(seq, len(seq) // self.block_size - 1)

    # ------------------------------------------------------------------ publish after compute
    def _record_completed_block_hash(self, seq, block_idx: int, *, publish: Optional[bool] = None):
        if not 0 <= block_idx < len(seq.block_table):
            return None
        if seq.block_has_unmaterialized_device_tokens(block_idx):
            return None
        bs = self.block_size
        toks = seq.token_ids[block_idx * bs:(block_idx + 1) * bs]
        if len(toks) != bs:
            return None
        blk = self.blocks[seq.block_table[block_idx]]
        do_publish = seq.prefix_cache_enabled if publish is None else bool(publish)
        if blk.hash == NO_HASH:
            prev = self.blocks[seq.block_table[block_idx - 1]].hash if block_idx > 0 else NO_HASH
            blk.update(self.compute_hash(toks, prev), toks)
        if do_publish:
            self.hash_to_block_id[blk.hash] = blk.block_id
        return blk.hash

    def record_computed_prefix(self, seq, upto_tokens: int, *, publish: bool):
        """Record digests of the full prompt blocks below `upto_tokens`; return the last one's
        digest when `upto_tokens` is a positive multiple of the block size, else None."""
        upto = max(0, min(int(upto_tokens), int(seq.num_prompt_tokens)))
        full = upto // self.block_size
        last = None
        for idx in range(full):
            last = self._record_completed_block_hash(seq, idx, publish=publish)
        return last if (upto > 0 and upto % self.block_size == 0) else None

    def publish_computed_prefix(self, seq, upto_tokens: int):
        return self.record_computed_prefix(seq, upto_tokens, publish=True)

    # ------------------------------------------------------------------ diagnostics
    def stats(self) -> dict:
        return {"total_blocks": len(self.blocks), "free_blocks": len(self.free_block_ids),
                "used_blocks": len(self.used_block_ids)}

    def snapshot(self, seqs=None) -> BlockTables:
        return BlockTables(tables=[list(s.block_table) for s in seqs] if seqs is not None else [],
                           ref_counts=[b.ref_count for b in self.blocks],
                           hashes=[b.hash for b in self.blocks])
