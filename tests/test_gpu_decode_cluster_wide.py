"""The cluster form for rows of 2 - 4 query tokens against the streaming forms: both tile counts, block edges of a row, every
cluster size, tokens that see nothing, and a block id outside the pool."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE, decode_case, to_torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [2, 3, 4])
@pytest.mark.parametrize("rows,width", [(3, 2), (3, 5), (2, 20), (1, 80), (40, 9), (150, 6)])
def test_equals_the_streaming_form(tokens, rows, width):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    span = width * BS
    edges = [n for n in (1, 15, 16, 17, 31, 33, span - 16, span - 1, span, 0) if n <= span]
    lens = np.asarray([edges[(i + tokens) % len(edges)] for i in range(rows)], np.int32)
    nblk = int((-(-lens // BS)).sum()) + 9
    rng = np.random.default_rng(rows + tokens)
    c = decode_case(tokens, nblk, rows, 1, 1, width=width)
    perm, o = rng.permutation(nblk), 0
    tables = np.zeros((rows, width), np.int32)
    for b, n in enumerate(-(-lens // BS)):
        tables[b, :n] = perm[o:o + n]
        o += n
    k, v = (to_torch(c[n])[0].to(torch.bfloat16) for n in ("k_cache", "v_cache"))
    for t in (k, v):  # what lies behind a row's last key must not reach the result
        for b, n in enumerate(lens):
            if n % BS:
                t[int(tables[b, n // BS]), n % BS:] = 1000.0
    q = to_torch(rng.standard_normal((rows, tokens, 8, 256)).astype(np.float32)).to(torch.bfloat16)
    pos = lens[:, None] - tokens + np.arange(tokens)[None]  # short rows: the first tokens see nothing
    pos[::3, -1] = -1                                       # padding
    args = q, k, v, to_torch(tables), to_torch(lens)
    for p in (to_torch(pos.astype(np.int32)), None):
        got = K.paged_decode_attention_wide(*args, p, SCALE, form=3)
        ref = K.paged_decode_attention_wide(*args, p, SCALE, form=2)
        assert float((got - ref).abs().max()) <= 2e-3
        assert not got[args[4] == 0].any()
        if p is not None:
            assert not got[p < 0].any()


def test_a_bad_block_is_flagged_and_left_out(monkeypatch):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    c = decode_case(3, 8, 2, 1, 1, width=4)
    k, v = (to_torch(c[n])[0].to(torch.bfloat16) for n in ("k_cache", "v_cache"))
    q = torch.randn((2, 3, 8, 256), device=k.device).to(torch.bfloat16)
    lens = to_torch(np.asarray([40, 64], np.int32))
    tables = to_torch(np.asarray([[0, 1, 8, 0], [3, 4, 5, 6]], np.int32))  # the pool ends at 7
    with pytest.raises(K.DeviceStatusError):
        K.paged_decode_attention_wide(q, k, v, tables, lens, None, SCALE, form=3)
    monkeypatch.setenv("NVJ_CHECK_STATUS", "0")
    got = K.paged_decode_attention_wide(q, k, v, tables, lens, None, SCALE, form=3)
    with pytest.raises(K.DeviceStatusError):
        K.check_device_status()
    good = to_torch(np.asarray([[0, 1, 7, 0], [3, 4, 5, 6]], np.int32))
    ref = K.paged_decode_attention_wide(q, k, v, good, torch.tensor([32, 64], dtype=torch.int32, device="cuda"), None, SCALE, form=2)
    assert float((got - ref).abs().max()) <= 2e-3


def _batch(seed, rows, width, tokens, kind="plain"):
    """Rows of 4 keys per table block up to the whole table over scattered blocks, their last `tokens` tokens as queries."""
    g, rng = torch.Generator(device="cuda").manual_seed(seed), np.random.default_rng(seed)
    lens = np.maximum(rng.integers(4 * width, BS * width + 1, rows), tokens)
    need = -(-lens // BS)
    pool = int(need.sum())
    k, v = (torch.randn((pool, BS, 2, 256), generator=g, device="cuda") for _ in range(2))
    tables = torch.zeros((rows, width), dtype=torch.int32, device="cuda")
    tables[torch.arange(width, device="cuda")[None] < to_torch(need)[:, None]] = torch.randperm(pool, generator=g, device="cuda").to(torch.int32)
    q = torch.randn((rows, tokens, 8, 256), generator=g, device="cuda") * (6 if kind == "peaked" else 1)
    lens = to_torch(lens.astype(np.int32))
    pos = (lens[:, None] - tokens + torch.arange(tokens, dtype=torch.int32, device="cuda")).contiguous()
    return q.to(torch.bfloat16), k.to(torch.bfloat16), (v + (3 if kind == "offset" else 0)).to(torch.bfloat16), tables, lens, pos


def _in_64_bits(q, k, v, tables, lens, pos):
    keys, values = (t[tables.long()].reshape(len(lens), -1, 2, 256).double() for t in (k, v))
    x = q.double().view(len(lens), -1, 2, 4, 256)
    s = torch.einsum("bwhgd,bkhd->bwhgk", x, keys) * SCALE
    see = (torch.arange(s.shape[-1], device="cuda") <= pos[..., None])[:, :, None, None]
    return torch.einsum("bwhgk,bkhd->bwhgd", s.masked_fill(~see, -float("inf")).softmax(-1), values).reshape(len(lens), -1)


@pytest.mark.parametrize("rows,width,tokens", [(600, 8, 2), (1100, 12, 3), (3200, 4, 4)])
@pytest.mark.parametrize("kind", ["plain", "peaked", "offset"])
def test_many_short_rows_are_as_near_64_bits_as_on_mma_sync(rows, width, tokens, kind):
    """Beyond the blocks that go to tcgen05 the mma.sync form is what a row would run on otherwise.  Both round as many partial sums, in
    another order, so their errors differ by chance alone: over 600 rows and more by less than 1 in 100 (3 allowed; one sum of
    all blocks of a row is 8 in 100 and more behind)."""
    from nano_vllm_jax_b200.kernels import paged_kv as K
    args = _batch(5, rows, width, tokens, kind)
    want = _in_64_bits(*args)
    off = [float((K.paged_decode_attention_wide(*args, SCALE, form=f).view_as(want) - want).norm()) for f in (0, 1)]
    assert off[0] <= 1.03 * off[1]


# both sides of every end of the rule for many short rows: 2 tokens at 24 and 25 blocks, 3 and 4 tokens at 16 blocks and at 12288 blocks
# of table in all; and of the rule for few blocks per CTA (the forms: 1 mma.sync, 2 tcgen05, 3 clusters)
@pytest.mark.parametrize("tokens,rows,width,form", [(2, 100, 25, 3), (2, 400, 25, 3), (2, 401, 25, 1), (2, 401, 24, 3), (2, 2000, 24, 3), (2, 2000, 25, 1),
                                                    (2, 130, 30, 3), (2, 160, 25, 3), (2, 160, 26, 1), (3, 768, 16, 3), (3, 769, 16, 1),
                                                    (4, 3072, 4, 3), (4, 3073, 4, 1), (4, 200, 17, 2), (3, 64, 40, 3), (3, 64, 43, 2)])
def test_the_form_that_the_rule_takes(tokens, rows, width, form):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are drawn for 148 SMs")
    args = _batch(rows + width, rows, width, tokens)
    auto, *by_form = (K.paged_decode_attention_wide(*args, SCALE, form=f) for f in (0, 1, 2, 3))
    assert [f for f, out in enumerate(by_form, 1) if torch.equal(out, auto)] == [form]  # (no two forms sum in one order)
