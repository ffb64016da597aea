"""Rows of 2 - 16 query tokens on tcgen05, on clusters (a narrow table) and on ranges (the same rows under a table too wide for
them, or too many rows), against attention in 64 bits: edges of the 16-key blocks and 128-key tiles, every cluster size, rows without
keys, what lies behind a row's last key, rows cut over several ranges."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE, to_torch

pytestmark = pytest.mark.gpu


def _batch(lens, width, tokens, seed, behind):
    g, rng = torch.Generator(device="cuda").manual_seed(seed), np.random.default_rng(seed)
    need = -(-lens // BS)
    pool = int(need.sum()) + 5
    k, v = (torch.randn((pool, BS, 2, 256), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    tables, ids, o = np.zeros((len(lens), width), np.int32), rng.permutation(pool), 0
    for b, n in enumerate(need):
        tables[b, :n] = ids[o:o + n]
        o += n
        if lens[b] % BS:
            for t in (k, v):
                t[int(tables[b, n - 1]), lens[b] % BS:] = behind
    q = torch.randn((len(lens), tokens, 8, 256), generator=g, device="cuda").to(torch.bfloat16)
    pos = lens[:, None] - tokens + np.arange(tokens)[None]  # short rows: the first tokens see nothing
    pos[1::3, -1] = -1                                      # padding
    return q, k, v, to_torch(tables), to_torch(lens.astype(np.int32)), to_torch(pos.astype(np.int32))


def _in_64_bits(q, k, v, tables, lens, pos):
    out = torch.zeros(q.shape[0], q.shape[1], 8 * 256, dtype=torch.float64, device="cuda")
    for b, n in enumerate(lens.tolist()):
        ids = tables[b, :-(-n // BS)].long()
        keys, values = (t[ids].reshape(-1, 2, 256)[:n].double().repeat_interleave(4, 1) for t in (k, v))
        s = torch.einsum("whd,khd->whk", q[b].double(), keys) * SCALE
        see = torch.arange(n, device="cuda")[None] <= pos[b, :, None]
        w = s.masked_fill(~see[:, None], -float("inf")).softmax(-1).nan_to_num(0.0)  # (a token that sees nothing: zeros)
        out[b] = torch.einsum("whk,khd->whd", w, values).reshape(q.shape[1], -1)
    return out


# rows x table width pick clusters of 1 (both), 16, 16, 10, 6, 2, 1 and 1 CTAs; 75 rows and more do not fit
@pytest.mark.parametrize("rows,width", [(1, 4), (1, 40), (3, 200), (4, 60), (8, 150), (36, 20), (48, 11), (74, 9), (75, 9), (150, 6)])
@pytest.mark.parametrize("tokens", [2, 5, 8, 9, 16])
def test_on_clusters_and_on_ranges(tokens, rows, width):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    span = width * BS
    edges = [n for n in (span, 1, 15, 16, 17, 0, 127, 128, 129, span - 16, span - 1, 257, 640) if n <= span]
    lens = np.asarray([edges[(i + tokens) % len(edges)] if rows > 1 else span - tokens for i in range(rows)])
    # up to 8 tokens what lies behind the last key reaches nothing; a weight of zero times a value does, where the rows are the tile's
    q, k, v, tables, lens, pos = _batch(lens, width, tokens, rows + tokens, float("nan") if tokens <= 8 else 1000.0)
    want = _in_64_bits(q, k, v, tables, lens, pos)
    wide = torch.zeros(rows, 801, dtype=torch.int32, device="cuda")
    wide[:, :width] = tables
    for t in (tables, wide):
        got = K.paged_decode_attention_wide(q, k, v, t, lens, pos, SCALE, form=2).view_as(want)
        assert float((got - want).abs().max()) <= 2e-3
        assert not got[lens == 0].any() and not got[pos < 0].any()


@pytest.mark.parametrize("tokens", [3, 6, 8, 12])
@pytest.mark.parametrize("lens", [[4000] * 3 + [1, 900, 0, 130], [30000], [7, 20000, 7, 9000], [600 + 37 * i for i in range(90)]])
def test_rows_cut_over_ranges(tokens, lens):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    lens = np.asarray(lens)
    q, k, v, tables, lens, pos = _batch(lens, max(900, -(-int(lens.max()) // BS)), tokens, len(lens) + tokens, 1000.0)
    want = _in_64_bits(q, k, v, tables, lens, pos)
    got = K.paged_decode_attention_wide(q, k, v, tables, lens, pos, SCALE, form=2)
    assert float((got.view_as(want) - want).abs().max()) <= 2e-3
    assert torch.equal(got, K.paged_decode_attention_wide(q, k, v, tables, lens, pos, SCALE, form=2))  # the fold's order is fixed


@pytest.mark.parametrize("tokens", [5, 9])
@pytest.mark.parametrize("width", [20, 801])
def test_a_bad_block_is_flagged(tokens, width, monkeypatch):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    args = list(_batch(np.asarray([300, 200]), width, tokens, 3, 1000.0))
    good = K.paged_decode_attention_wide(*args, SCALE, form=2)
    args[3][0, 5] = args[1].shape[0]
    monkeypatch.setenv("NVJ_CHECK_STATUS", "0")
    bad = K.paged_decode_attention_wide(*args, SCALE, form=2)
    with pytest.raises(K.DeviceStatusError):
        K.check_device_status()
    assert torch.equal(bad[1], good[1]) and torch.isfinite(bad).all()
