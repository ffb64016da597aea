"""The cluster form of the decode kernel against the generic one: block, unit and warp boundaries of a row, every cluster
size, every cache and query dtype, both forms of the fused append, and a block id outside the pool."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE, bits, decode_case, to_numpy, to_torch

pytestmark = pytest.mark.gpu

TIGHT = {torch.bfloat16: 2e-3, torch.float16: 5e-4, torch.float32: 2e-5}


def _case(seed, lens, width, dtype):
    c = decode_case(seed, int(sum(-(-n // BS) for n in lens)) + 9, len(lens), 1, 1, width=width)
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens, np.int32)
    perm = rng.permutation(c["k_cache"].shape[1])
    tables, o = np.zeros((len(lens), width), np.int32), 0
    for b, n in enumerate(-(-lens // BS)):
        tables[b, :n] = perm[o:o + n]
        o += n
    k, v = (to_torch(c[n]).to(dtype) for n in ("k_cache", "v_cache"))
    for t in (k, v):  # what lies behind a row's last key must not reach the result
        for b, n in enumerate(lens):
            if n % BS:
                t[0, int(tables[b, n // BS]), n % BS:] = float("nan")
    return k, v, to_torch(tables), to_torch(lens), c


# rows x table width (in blocks) pick the cluster size: 1, 3, 5, 10 and 16 CTAs per row and KV head in small batches, then 7, 5
# and 3, then 3 and 2 CTAs per row for both heads
@pytest.mark.parametrize("rows,width", [(3, 4), (3, 9), (3, 20), (3, 40), (2, 80), (28, 30), (40, 24), (60, 14), (130, 9), (150, 6)])
@pytest.mark.parametrize("cache,query", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16), (torch.float32, torch.float32),
                                         (torch.float16, torch.float32), (torch.float32, torch.bfloat16)])
def test_cluster_decode_equals_the_generic_kernel(rows, width, cache, query):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    span = width * BS
    edges = [n for n in (1, 3, 4, 15, 16, 17, 63, 64, 65, span - 16, span - 1, span, 0) if n <= span]
    k, v, tables, lens, c = _case(rows + width, [edges[i % len(edges)] for i in range(rows)], width, cache)
    q = to_torch(c["q"][:, 0]).to(query).contiguous()
    got = K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE, variant=4)
    ref = K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE, variant=1)
    assert float((got - ref).abs().max()) <= TIGHT[cache]
    assert not got[lens == 0].any()


@pytest.mark.parametrize("pre_append", [False, True])
@pytest.mark.parametrize("cache", [torch.bfloat16, torch.float16, torch.float32])
def test_cluster_decode_with_the_fused_append(cache, pre_append):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    lens = [1, 16, 17, 33, 0, 144, 129]
    k, v, tables, t_lens, c = _case(5, lens, 9, cache)
    q, nk, nv = (to_torch(c[n]).to(cache) for n in ("q", "new_k", "new_v"))
    pos = (t_lens - 1).clamp(min=0).view(-1, 1).contiguous()
    k2, v2 = k.clone(), v.clone()
    for b, n in enumerate(lens):
        if n:
            block, off = int(tables[b, (n - 1) // BS]), (n - 1) % BS
            k2[0, block, off], v2[0, block, off] = nk[b, 0], nv[b, 0]
    ref = K.paged_decode_attention(q[:, 0].contiguous(), k2[0], v2[0], tables, t_lens, SCALE, variant=1)
    before = torch.where(t_lens > 0, t_lens - 1, t_lens)
    if pre_append:  # a row of length 1 would be inactive before its first token: leave it out of the comparison
        ref = ref.clone()
        ref[0] = 0
        k2[0, int(tables[0, 0]), 0], v2[0, int(tables[0, 0]), 0] = k[0, int(tables[0, 0]), 0], v[0, int(tables[0, 0]), 0]
    out, k, v = K.paged_decode_attention_with_kv_append(q, nk, nv, k, v, tables, before if pre_append else t_lens,
                                                        None if pre_append else pos, 0, BS, SCALE, 4, variant=4)
    assert float((out.view(7, 8, 256) - ref).abs().max()) <= TIGHT[cache]
    for a, b in ((k, k2), (v, v2)):
        np.testing.assert_array_equal(bits(to_numpy(a)), bits(to_numpy(b)))


def test_cluster_decode_flags_a_bad_block_and_leaves_its_keys_out(monkeypatch):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    k, v, tables, lens, c = _case(8, [200, 90], 13, torch.bfloat16)
    q = to_torch(c["q"][:, 0]).contiguous()
    bad = tables.clone()
    bad[0, 12] = k.shape[1]  # the row's last block: the result is the row without it
    with pytest.raises(K.DeviceStatusError):
        K.paged_decode_attention(q, k[0], v[0], bad, lens, SCALE, variant=4)
    monkeypatch.setenv("NVJ_CHECK_STATUS", "0")
    got = K.paged_decode_attention(q, k[0], v[0], bad, lens, SCALE, variant=4)
    ref = K.paged_decode_attention(q, k[0], v[0], tables, torch.tensor([192, 90], dtype=torch.int32, device="cuda"), SCALE, variant=1)
    with pytest.raises(K.DeviceStatusError):
        K.check_device_status()
    assert float((got - ref).abs().max()) <= 2e-3


# the launched form's own numbers decide (CTAs per row, blocks per walking warp, how often the CTAs fill their places); rows far
# shorter than the table, the case a padded table makes, in every form: 5, 8, 6 and 6 CTAs per row for both heads, 8 per head
@pytest.mark.parametrize("rows,width,pays", [(68, 200, True), (96, 263, True), (130, 100, True), (256, 263, True), (67, 384, False),
                                             (160, 144, False), (123, 263, False), (256, 400, False), (70000, 4, False)])
def test_short_rows_under_a_wide_table(rows, width, pays):
    from nano_vllm_jax_b200 import _lib
    from nano_vllm_jax_b200.kernels import paged_kv as K
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert bool(_lib.load().nvj_paged_decode_on_clusters(rows, width)) == pays
    if rows > 1000:
        return
    lens = [1 + (37 * i) % 150 for i in range(rows - 2)] + [0, width * BS - 5]
    k, v, tables, lens, c = _case(rows, lens, width, torch.bfloat16)
    k, v = k.nan_to_num(), v.nan_to_num()  # (what the streaming kernel reads behind a row's last key must be finite)
    q = to_torch(c["q"][:, 0]).contiguous()
    ref = K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE, variant=1)
    for variant in (0, 4):
        assert float((K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE, variant=variant) - ref).abs().max()) <= 2e-3


@pytest.mark.parametrize("rows,width", [(37, 100), (38, 100), (150, 60)])  # 8, 4 and 4 CTAs per row and head
@pytest.mark.parametrize("cache,query", [(torch.float32, torch.float32), (torch.float16, torch.float32)])
def test_short_rows_under_a_wide_table_on_the_cuda_cores(rows, width, cache, query):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    lens = [1 + (37 * i) % 150 for i in range(rows - 2)] + [0, width * BS - 5]
    k, v, tables, lens, c = _case(rows, lens, width, cache)
    q = to_torch(c["q"][:, 0]).to(query).contiguous()
    ref = K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE, variant=1)
    got = K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE)
    assert float((got - ref).abs().max()) <= TIGHT[cache]


# eight CTAs and more per row and head, all resident: up to 16 blocks per walker; 32 rows' eight are not
@pytest.mark.parametrize("rows,width,pays", [(16, 512, True), (24, 512, True), (24, 520, False), (32, 400, False), (8, 2048, False)])
def test_few_rows_of_many_blocks(rows, width, pays):
    from nano_vllm_jax_b200 import _lib
    from nano_vllm_jax_b200.kernels import paged_kv as K
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert bool(_lib.load().nvj_paged_decode_on_clusters(rows, width)) == pays
    if rows * width > 8192:
        return
    lens = [1 + (1037 * i) % (width * BS) for i in range(rows - 1)] + [width * BS]
    k, v, tables, lens, c = _case(rows, lens, width, torch.bfloat16)
    q = to_torch(c["q"][:, 0]).contiguous()
    ref = K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE, variant=1)
    assert float((K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE) - ref).abs().max()) <= 2e-3


# What the kernel looks at ahead of its wait is a hint: here the kernel in front changes the lengths (rows gain a key, some a block)
# and the tables hold ids outside the pool behind the last block.  CTAs with the hint and, beyond three to an SM, without it.
@pytest.mark.parametrize("rows,width", [(3, 5), (48, 20), (300, 6)])
def test_lengths_that_the_kernel_in_front_changes(rows, width, monkeypatch):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    monkeypatch.setenv("NVJ_CHECK_STATUS", "1")  # nothing may be flagged
    before = [(0, 15, 16, 47, width * BS - 1, 33)[i % 6] for i in range(rows)]
    k, v, tables, lens, c = _case(rows, [n + 1 if n else 0 for n in before], width, torch.bfloat16)
    used = torch.arange(width, device="cuda")[None] * BS < lens[:, None]
    tables = torch.where(used, tables, torch.full_like(tables, k.shape[1] + 7))
    q = to_torch(c["q"][:, 0]).contiguous()
    ref = K.paged_decode_attention(q, k[0], v[0], tables, lens, SCALE, variant=1)
    x = torch.randn(rows, 2048, device="cuda")
    for _ in range(3):
        now = torch.tensor(before, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        K.row_argmax(x, advance=(now, None, width, BS))
        got = K.paged_decode_attention(q, k[0], v[0], tables, now, SCALE, variant=4)
        assert torch.equal(now, lens)
        assert float((got - ref).abs().max()) <= 2e-3


# the warp that stores the new row is the one whose block it falls into: among its first 32 blocks or behind them, in a block that the
# row does not attend, and in the last one of the table
@pytest.mark.parametrize("cache", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("lens,at", [([33605, 90, 20], [33604, 89, 19]), ([100, 1, 200], [170, 63, 991]), ([16, 32, 48], [16, 31, 300])])
def test_cluster_decode_appends_wherever_the_position_lies(cache, lens, at):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    width = max(max(lens), max(at) + 1) // BS + 1
    g = torch.Generator(device="cuda").manual_seed(sum(at))
    k, v = (torch.randn((1, 3 * width + 4, BS, 2, 256), generator=g, device="cuda").to(cache) for _ in range(2))
    tables = torch.randperm(3 * width + 4, generator=g, device="cuda").to(torch.int32)[:3 * width].view(3, width).contiguous()
    t_lens, pos = torch.tensor(lens, dtype=torch.int32, device="cuda"), torch.tensor(at, dtype=torch.int32, device="cuda").view(3, 1)
    q, nk, nv = (torch.randn((3, 1, h, 256), generator=g, device="cuda").to(cache) for h in (8, 2, 2))
    k2, v2 = k.clone(), v.clone()
    for b, p in enumerate(at):
        k2[0, int(tables[b, p // BS]), p % BS], v2[0, int(tables[b, p // BS]), p % BS] = nk[b, 0], nv[b, 0]
    ref = K.paged_decode_attention(q[:, 0].contiguous(), k2[0], v2[0], tables, t_lens, SCALE, variant=1)
    out, k, v = K.paged_decode_attention_with_kv_append(q, nk, nv, k, v, tables, t_lens, pos, 0, BS, SCALE, 4, variant=4)
    assert float((out.view(3, 8, 256) - ref).abs().max()) <= TIGHT[cache]
    for a, b in ((k, k2), (v, v2)):
        np.testing.assert_array_equal(bits(to_numpy(a)), bits(to_numpy(b)))
