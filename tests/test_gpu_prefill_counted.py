"""Packed prefill launched for exactly the tiles that the host counted: the same rows as without the count, padding zeroed,
and a count that is too small flagged instead of passing for a result."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE, to_torch

pytestmark = pytest.mark.gpu


def _batch(qlens, cached, pad, seed):
    rng = np.random.default_rng(seed)
    lens = np.array([q + c for q, c in zip(qlens, cached)], np.int32)
    need = -(-lens // BS)
    tables, o = np.zeros((len(qlens), int(need.max())), np.int32), 0
    perm = rng.permutation(int(need.sum()) + 8)
    for r, n in enumerate(need):
        tables[r, :n] = perm[o:o + n]
        o += n
    pos = np.concatenate([np.arange(c, c + q) for q, c in zip(qlens, cached)] + [np.zeros(pad, int)]).astype(np.int32)[None]
    rid = np.concatenate([np.repeat(np.arange(len(qlens)), qlens), np.zeros(pad, int)]).astype(np.int32)[None]
    g = torch.Generator(device="cuda").manual_seed(seed)
    cache = [torch.randn((1, int(need.sum()) + 8, BS, 2, 256), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    q = torch.randn((1, pos.shape[1], 8, 256), generator=g, device="cuda").to(torch.bfloat16)
    return q, cache, to_torch(tables), to_torch(lens), to_torch(pos), to_torch(rid), to_torch(np.cumsum([0] + list(qlens)).astype(np.int32))


@pytest.mark.parametrize("qlens,cached,pad", [
    ((64,), (0,), 0), ((65, 2), (0, 70), 3), ((63, 64, 128), (5, 0, 300), 0),       # no decode rows: key ranges may be split
    ((1, 1, 130, 1, 40), (40, 700, 0, 3, 90), 7), ((1,) * 40 + (2,), (33,) * 40 + (0,), 0),  # decode rows beside the tiles
    ((1,) * 30 + (300,) * 8, (500,) * 30 + (0,) * 8, 0),                            # ... and tiles on every SM
])
def test_counted_launch_equals_the_uncounted_one(qlens, cached, pad):
    from nano_vllm_jax_b200 import kv_cache as kvc
    q, (k, v), tables, lens, pos, rid, qsl = _batch(qlens, cached, pad, len(qlens) + pad)
    singles, pairs = sum(n == 1 for n in qlens), sum(-(-n // 64) for n in qlens if n > 1)

    def run(count):
        return kvc.paged_attention_prefill_packed(q, k, v, tables, lens, pos, rid, qsl, BS, SCALE, 4, out_dtype=torch.float32,
                                                  num_decode_rows=singles, query_tile_pairs=count)

    out, ref = run(pairs), run(None)
    assert float((out - ref).abs().max()) <= 2e-3
    assert not out[0, sum(qlens):].any() and not torch.isnan(out).any()


def test_a_count_that_is_too_small_is_flagged(monkeypatch):
    from nano_vllm_jax_b200 import kv_cache as kvc
    from nano_vllm_jax_b200.kernels.paged_kv import DeviceStatusError
    q, (k, v), tables, lens, pos, rid, qsl = _batch((200, 90), (0, 0), 0, 3)
    with pytest.raises(DeviceStatusError):
        kvc.paged_attention_prefill_packed(q, k, v, tables, lens, pos, rid, qsl, BS, SCALE, 4, out_dtype=torch.float32,
                                           num_decode_rows=0, query_tile_pairs=3)


# key ranges around where a pair is split (5, 6, 7 tiles of 64 keys), long ones in 4, 3 and 2 pieces as the batch leaves room, a row
# of each kind in one launch, rows without keys, and a batch whose pairs do not all fit beside each other in clusters of four
@pytest.mark.parametrize("qlens,cached,pad", [
    ((2,), (5 * 64 - 3,), 1), ((64,), (5 * 64,), 0), ((33, 64), (6 * 64, 6 * 64 + 1), 5), ((2, 130, 70, 5), (0, 1500, 300, 900), 9),
    ((64,) * 6, (1000, 0, 350, 330, 2000, 64), 0), ((64,) * 8, (700,) * 8, 3), ((300, 200, 90), (512, 1024, 0), 0), ((64,) * 20, (800,) * 20, 0),
])
def test_split_key_ranges_equal_the_kernel_that_never_splits(qlens, cached, pad):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    q, (k, v), tables, lens, pos, rid, qsl = _batch(qlens, cached, pad, sum(qlens))
    pairs = sum(-(-n // 64) for n in qlens)
    args = (q, k[0], v[0], tables, lens, pos, qsl, BS, SCALE, 4)
    ref = K.packed_paged_prefill_attention(*args, variant=3, num_decode_rows=0)
    for count in (pairs, None):
        out = K.packed_paged_prefill_attention(*args, variant=4, num_decode_rows=0, query_tile_pairs=count)
        assert float((out - ref).abs().max()) <= 2e-3 and not out[0, sum(qlens):].any()


@pytest.mark.parametrize("route", ["python", "extension"])
def test_key_ranges_stay_whole_where_the_caller_says_so(monkeypatch, route):
    """NVJ_PREFILL_KEY_SPLITS=0: bit for bit what the same rows give beside a decode row, whose batch is never split."""
    from nano_vllm_jax_b200 import kv_cache as kvc
    from nano_vllm_jax_b200.kernels import paged_kv as K
    q, (k, v), tables, lens, pos, rid, qsl = _batch((130, 64, 1), (1500, 700, 20), 0, 9)

    def run(rows):
        n = int(qsl[rows])
        if route == "python":
            return K.packed_paged_prefill_attention(q[:, :n], k[0], v[0], tables[:rows], lens[:rows], pos[:, :n], qsl[: rows + 1], BS, SCALE, 4,
                                                    variant=4, num_decode_rows=rows - 2)[0, :194]
        return kvc.paged_attention_prefill_packed(q[:, :n], k, v, tables[:rows], lens[:rows], pos[:, :n], rid[:, :n], qsl[: rows + 1], BS, SCALE,
                                                  4, out_dtype=torch.float32, num_decode_rows=rows - 2)[0, :194]

    whole, split = run(3), run(2)
    assert not torch.equal(whole, split) and float((whole - split).abs().max()) <= 2e-3
    monkeypatch.setenv("NVJ_PREFILL_KEY_SPLITS", "0")
    assert torch.equal(run(2).view(torch.int32), whole.view(torch.int32))


# 1 - 10 key tiles (one and two of them per softmax group, odd and even numbers), key ranges whole and split, splits that begin behind the
# row's first 128 blocks; keys that grow by more than the rescale gap from every tile to the next, shrink, or neither
@pytest.mark.parametrize("growth", [0.0, 3.0, -3.0])
@pytest.mark.parametrize("qlens,cached", [((64,), (0,)), ((40, 64, 2), (64, 128, 190)), ((64, 33), (250, 300)), ((64,), (576,)), ((17,), (2900,)),
                                          ((64,) * 24, (37,) * 12 + (290,) * 12)])
def test_tiles_taken_in_turn_follow_the_rows_maximum(qlens, cached, growth, monkeypatch):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    q, (k, v), tables, lens, pos, rid, qsl = _batch(qlens, cached, 0, sum(qlens))
    for r, n in enumerate(lens.tolist()):
        blocks = tables[r, :-(-n // BS)].long()
        tile = torch.arange(len(blocks), device="cuda") // 4
        size = 1 + abs(growth) * (tile if growth > 0 else tile.max() - tile).clamp(max=10)
        k[0, blocks] = (k[0, blocks].float() * size[:, None, None, None]).to(torch.bfloat16)
    ref = torch.zeros(q.shape[1], 8, 256, dtype=torch.float64, device="cuda")
    for r, n in enumerate(lens.tolist()):
        a, b = qsl[r].item(), qsl[r + 1].item()
        keys, values = (c[0, tables[r].long()].double().reshape(-1, 2, 256)[:n].repeat_interleave(4, 1) for c in (k, v))
        s = torch.einsum("qhd,khd->hqk", q[0, a:b].double(), keys) * SCALE
        s.masked_fill_(torch.arange(n, device="cuda") > pos[0, a:b, None], float("-inf"))
        ref[a:b] = torch.einsum("hqk,khd->qhd", s.softmax(-1), values)
    args = (q, k[0], v[0], tables, lens, pos, qsl, BS, SCALE, 4)
    for splits in ("1", "0"):
        monkeypatch.setenv("NVJ_PREFILL_KEY_SPLITS", splits)
        out = K.packed_paged_prefill_attention(*args, num_decode_rows=0, query_tile_pairs=sum(-(-n // 64) for n in qlens))
        # scores of up to ~130 natural units carry 2^-21 of rounding of their 256 products' sum: 1e-4 of a weight, values below 6
        assert float((out[0].reshape(-1, 8, 256).double() - ref).abs().max()) <= 2e-3
