"""The host module's calls against the Python route: the same numbers from operands it declines (strided, int64) as from
those it takes, slots made inside the append equal the slot mapping's, lengths capped inside the kernel equal lengths
clipped in front of it."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE, bits, decode_case, to_numpy, to_torch

pytestmark = pytest.mark.gpu


def _strided(t):
    """The same values behind a layout that the host module declines."""
    return torch.stack([t, t], -1)[..., 0]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("rows", [1, 5])
def test_fused_decode_takes_both_routes_alike(rows, dtype):
    from nano_vllm_jax_b200.backends import B200Backend
    from nano_vllm_jax_b200.kernels import paged_kv as K
    from nano_vllm_jax_b200.kv_cache import KVCacheStorage
    c = decode_case(3 + rows, 200, rows, 1, 300)
    got = []
    for odd in (False, True):
        cache = KVCacheStorage(to_torch(c["k_cache"]).to(dtype), to_torch(c["v_cache"]).to(dtype))
        args = [to_torch(c[n]).to(dtype) for n in ("q", "new_k", "new_v")]
        tables, lens, pos = (to_torch(c[n]) for n in ("tables", "seq_lens", "positions"))
        if odd:
            args, lens, tables = [_strided(t) for t in args], lens.to(torch.int64), _strided(tables)
            assert K.host().fused_decode(*args, cache.k_cache, cache.v_cache, tables, lens, pos, 0, BS, SCALE, 4, 0, None, None) is None
        be = B200Backend()
        md = be.build_attention_metadata(pos, tables, lens, BS, False)
        cache, out = be.write_kv_and_attention(0, *args, cache, md, BS, SCALE, 4, False)
        got.append((out, cache.k_cache, cache.v_cache))
    for a, b in zip(*got):
        assert a.dtype == b.dtype and a.shape == b.shape
        np.testing.assert_array_equal(bits(to_numpy(a)), bits(to_numpy(b)))


@pytest.mark.parametrize("width,max_kv_len", [(1, None), (1, 37), (3, None), (3, 48), (6, 100)])
def test_window_decode_equals_lengths_clipped_in_front(width, max_kv_len):
    from nano_vllm_jax_b200 import kv_cache as kvc
    from nano_vllm_jax_b200.kernels import paged_kv as K
    c = decode_case(11, 300, 7, width, 400, empty_rows=(2,))
    g = torch.Generator(device="cuda").manual_seed(1)
    q = torch.randn((7, width, 8, 256), generator=g, device="cuda").to(torch.bfloat16)
    k, v, tables, lens = (to_torch(c[n]) for n in ("k_cache", "v_cache", "tables", "seq_lens"))
    pos = (lens[:, None] - width - 3 + torch.arange(width, device="cuda")[None]).to(torch.int32).contiguous()  # some negative
    out = kvc.paged_attention_decode(q, k, v, tables, lens, BS, SCALE, 4, max_kv_len=max_kv_len, positions=pos, out_dtype=torch.float32)
    capped = lens.clamp(max=max_kv_len or tables.shape[1] * BS)
    if width == 1:
        ref = K.paged_decode_attention(q[:, 0].contiguous(), k[0], v[0], tables, torch.minimum(capped, pos[:, 0] + 1), SCALE)
    else:
        ref = K.paged_decode_attention_wide(q, k[0], v[0], tables, capped, pos, SCALE)
    assert torch.equal(out.reshape(-1), ref.reshape(-1))


@pytest.mark.parametrize("packed", [False, True])
def test_append_makes_the_slots_that_the_slot_mapping_has(packed):
    from nano_vllm_jax_b200.backends import B200Backend
    from nano_vllm_jax_b200.kv_cache import KVCacheStorage
    rng = np.random.default_rng(7)
    (rows, cols), pool = ((1, 40) if packed else (4, 9)), 64
    tables = to_torch(rng.permutation(pool)[:24].reshape(4, 6).astype(np.int32))
    places = rng.permutation(96)[: rows * cols] if packed else np.stack([rng.permutation(96)[:cols] for _ in range(rows)])
    pos = to_torch(places.reshape(rows, cols).astype(np.int32))
    rid = to_torch(np.sort(rng.integers(-1, 6, size=(1, cols))).astype(np.int32)) if packed else None  # clipped to the table's rows
    qsl = to_torch(np.array([0, 9, 18, 30, 35] if packed else [0, 9, 12, 21, 21], np.int32))
    new = [to_torch(rng.standard_normal((rows, cols, 2, 256)).astype(np.float32)) for _ in range(2)]
    got = []
    for read_first in (False, True):
        be = B200Backend()
        cache = KVCacheStorage(*(torch.zeros((2, pool, BS, 2, 256), dtype=torch.bfloat16, device="cuda") for _ in range(2)))
        md = be.build_attention_metadata(pos, tables, to_torch(np.full(4, 96, np.int32)), BS, True, query_start_loc=qsl, token_row_ids=rid)
        if read_first:
            assert md.slot_mapping.shape == pos.shape
        be.write_kv(1, *new, cache, md)
        got.append(cache)
    assert float(got[0].k_cache[1].float().abs().sum()) > 0 and not got[0].k_cache[0].any()
    assert torch.equal(got[0].k_cache, got[1].k_cache) and torch.equal(got[0].v_cache, got[1].v_cache)


@pytest.mark.parametrize("kind", ["decode", "prefill", "packed"])
@pytest.mark.parametrize("read_first", [False, True])
def test_when_the_slots_of_a_batch_are_made(kind, read_first):
    """A prefill's with its metadata, a decode batch's when they are read or appended to."""
    from nano_vllm_jax_b200.backends import B200Backend
    from nano_vllm_jax_b200.kv_cache import KVCacheStorage
    shape = (1, 6) if kind == "packed" else (2, 3)
    pos = torch.tensor([[0, 1, 2], [16, 17, 18]], dtype=torch.int32, device="cuda").view(shape)
    rid = torch.tensor([[0, 0, 0, 1, 1, 1]], dtype=torch.int32, device="cuda") if kind == "packed" else None
    tables = torch.tensor([[3, 1], [0, 2]], dtype=torch.int32, device="cuda")
    cache = KVCacheStorage(*(torch.zeros((1, 4, BS, 2, 256), dtype=torch.bfloat16, device="cuda") for _ in range(2)))
    be = B200Backend()
    md = be.build_attention_metadata(pos, tables, torch.tensor([3, 19], dtype=torch.int32, device="cuda"), BS, kind != "decode",
                                     query_start_loc=torch.tensor([0, 3, 6], dtype=torch.int32, device="cuda"), token_row_ids=rid)
    if read_first:
        md.slot_mapping
    pos += 4  # between the metadata and the append
    new = torch.ones((*shape, 2, 256), device="cuda", dtype=torch.bfloat16)
    be.write_kv(0, new, new, cache, md)
    moved = 4 if kind == "decode" and not read_first else 0
    assert cache.k_cache[0, :, :, 0, 0].nonzero().tolist() == [[b, t + moved] for b in (2, 3) for t in range(3)]


@pytest.mark.parametrize("packed", [False, True])
def test_the_mapped_append_writes_what_the_slot_mapping_says(packed):
    """nvj_kv_append_mapped against nvj_compute_slot_mapping + nvj_kv_append: row ids outside the table, rows shorter than the batch."""
    from nano_vllm_jax_b200 import _lib
    from nano_vllm_jax_b200.kernels import paged_kv as K
    lib, rng = _lib.load(), np.random.default_rng(8)
    (rows, cols), pool = ((1, 40) if packed else (4, 9)), 64
    tables = to_torch(rng.permutation(pool)[:24].reshape(4, 6).astype(np.int32))
    pos = to_torch(np.stack([rng.permutation(96)[:cols] for _ in range(rows)]).astype(np.int32))
    rid = to_torch(np.sort(rng.integers(-1, 6, size=(1, cols))).astype(np.int32)) if packed else None
    qsl = to_torch(np.array([0, 9, 18, 30, 35] if packed else [0, 9, 12, 21, 21], np.int32))
    new = [to_torch(rng.standard_normal((rows, cols, 2, 256)).astype(np.float32)).to(torch.bfloat16) for _ in range(2)]
    want, got = ([torch.zeros((pool, BS, 2, 256), dtype=torch.bfloat16, device="cuda") for _ in range(2)] for _ in range(2))
    K.kv_append_slots(*new, K.compute_slot_mapping(pos, tables, BS, rid), *want, query_start_loc=qsl, packed=packed)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = lib.nvj_kv_append_mapped(new[0].data_ptr(), new[1].data_ptr(), _lib.NVJ_BF16, pos.data_ptr(), tables.data_ptr(),
                                  rid.data_ptr() if packed else None, 4, 6, BS, qsl.data_ptr(), 4, int(packed), rows, cols,
                                  got[0].data_ptr(), got[1].data_ptr(), _lib.NVJ_BF16, pool * BS, 2, 256, status.data_ptr(),
                                  torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and int(status) == 0 and float(want[0].float().abs().sum()) > 0
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
