"""Rows of 9 - 16 query tokens on tcgen05, on ranges (query rows as the tile's rows) and on clusters: what the cache holds behind a row's last
key, infinities and NaN included, reaches nothing."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE
from test_gpu_decode_umma import _batch, _in_64_bits

pytestmark = pytest.mark.gpu


# last blocks of 1, 2, 15 and 16 keys, first, second and fourth of a tile of four, alone in it, and of rows cut over ranges
@pytest.mark.parametrize("behind", [float("nan"), float("inf")])
@pytest.mark.parametrize("tokens", [9, 12, 16])
@pytest.mark.parametrize("lens", [[17, 31, 32, 63, 1, 65, 0, 15, 49], [20000, 33, 9001], [601 + 37 * i for i in range(90)]])
def test_what_lies_behind_the_last_key_reaches_nothing(lens, tokens, behind):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    lens = np.asarray(lens)
    narrow = -(-int(lens.max()) // BS)
    q, k, v, tables, lens, pos = _batch(lens, narrow, tokens, len(lens) + tokens, behind)
    want = _in_64_bits(q, k, v, tables, lens, pos)
    wide = torch.zeros(len(lens), max(801, narrow), dtype=torch.int32, device="cuda")  # too wide for clusters
    wide[:, :narrow] = tables
    for t in (tables, wide):
        got = K.paged_decode_attention_wide(q, k, v, t, lens, pos, SCALE, form=2).view_as(want)
        assert float((got - want).abs().max()) <= 2e-3
