"""The streaming decode kernel against the generic one: block, walker and ring boundaries of a row and of a CTA's range, rows cut over
CTAs in one and in two levels, both forms of the fused append, whatever lies behind a row's last key, a block id outside the pool."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE, bits, to_numpy, to_torch
from test_gpu_decode_cluster import _case

pytestmark = pytest.mark.gpu

TIGHT = 2e-3  # bf16 operands, weights as two bf16 terms


# rows of 0 - 13 blocks share CTAs (a walker takes every fourth block, a ring holds 1.5); then rows cut over 3 - 10 CTAs, over more
# than 32 (folded in two levels), and more rows than a CTA's scan takes at a time
@pytest.mark.parametrize("lens", [[1, 15, 16, 17, 31, 33, 48, 49, 64, 65, 79, 0, 80, 81, 96, 97, 112, 113, 128, 129, 144, 145, 207, 208],
                                  [5], [16 * 6 * 3 + 1, 0, 16 * 6 * 10 - 1, 16 * 25], [16 * 6 * 40 + 3], [40 + (97 * i) % 300 for i in range(300)]])
def test_stream_decode_equals_the_generic_kernel(lens):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    k, v, tables, t_lens, c = _case(len(lens), lens, max(-(-n // BS) for n in lens) + 1, torch.bfloat16)
    q = to_torch(c["q"][:, 0]).contiguous()
    got = K.paged_decode_attention(q, k[0], v[0], tables, t_lens, SCALE, variant=3)
    ref = K.paged_decode_attention(q, k[0], v[0], tables, t_lens, SCALE, variant=1)
    assert float((got - ref).abs().max()) <= TIGHT
    assert not got[t_lens == 0].any()


@pytest.mark.parametrize("pre_append", [False, True])
def test_stream_decode_with_the_fused_append(pre_append):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    lens = [2, 16, 17, 33, 0, 144, 129, 16 * 6 * 5, 16 * 6 * 5 + 1]
    k, v, tables, t_lens, c = _case(5, lens, 32, torch.bfloat16)
    q, nk, nv = (to_torch(c[n]) for n in ("q", "new_k", "new_v"))
    pos = (t_lens - 1).clamp(min=0).view(-1, 1).contiguous()
    k2, v2 = k.clone(), v.clone()
    for b, n in enumerate(lens):
        if n:
            block, off = int(tables[b, (n - 1) // BS]), (n - 1) % BS
            k2[0, block, off], v2[0, block, off] = nk[b, 0], nv[b, 0]
    ref = K.paged_decode_attention(q[:, 0].contiguous(), k2[0], v2[0], tables, t_lens, SCALE, variant=1)
    before = torch.where(t_lens > 0, t_lens - 1, t_lens)
    out, k, v = K.paged_decode_attention_with_kv_append(q, nk, nv, k, v, tables, before if pre_append else t_lens,
                                                        None if pre_append else pos, 0, BS, SCALE, 4, variant=3)
    assert float((out.view(len(lens), 8, 256) - ref).abs().max()) <= TIGHT
    for a, b in ((k, k2), (v, v2)):
        np.testing.assert_array_equal(bits(to_numpy(a)), bits(to_numpy(b)))


@pytest.mark.parametrize("at", [0, 5, 12])  # the row's first, a middle and its last block
def test_stream_decode_flags_a_bad_block_and_leaves_its_keys_out(monkeypatch, at):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    k, v, tables, lens, c = _case(8, [208, 90], 13, torch.bfloat16)
    q = to_torch(c["q"][:, 0]).contiguous()
    bad = tables.clone()
    bad[0, at] = k.shape[1]
    without = tables.clone()  # the row without that block: the blocks behind it move up
    without[0, at:12] = tables[0, at + 1:]
    monkeypatch.setenv("NVJ_CHECK_STATUS", "0")
    got = K.paged_decode_attention(q, k[0], v[0], bad, lens, SCALE, variant=3)
    with pytest.raises(K.DeviceStatusError):
        K.check_device_status()
    ref = K.paged_decode_attention(q, k[0], v[0], without, torch.tensor([192, 90], dtype=torch.int32, device="cuda"), SCALE, variant=1)
    assert float((got - ref).abs().max()) <= TIGHT


# what a launch looks at ahead of its wait may still change: lengths and tables that a kernel in front replaces (values far outside
# the pool for a moment), batches of 1, 33 and 257 rows (one more than are looked through), and verification rows of 5 and 9 tokens
@pytest.mark.parametrize("rows,width", [(1, 1), (33, 1), (257, 1), (24, 5), (80, 5), (80, 9)])
def test_launches_that_follow_one_another_read_what_the_kernel_in_front_left(rows, width):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    g = torch.Generator(device="cuda").manual_seed(rows)
    blocks = 96 if rows == 1 else 24
    k, v = (torch.randn((1, 4096, BS, 2, 256), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    sets = [(torch.randint(width, blocks * BS + 1, (rows,), generator=g, device="cuda", dtype=torch.int32),
             torch.randint(0, 4096, (rows, blocks), generator=g, device="cuda", dtype=torch.int32)) for _ in range(3)]
    q = torch.randn((rows, width, 8, 256), generator=g, device="cuda").to(torch.bfloat16)

    def attend(lens, tables):
        if width == 1:
            return K.paged_decode_attention(q[:, 0].contiguous(), k[0], v[0], tables, lens, SCALE, variant=3)
        return K.paged_decode_attention_wide(q, k[0], v[0], tables, lens, None, SCALE, form=2)

    alone = []
    for s in sets:
        alone.append(attend(*s))
        torch.cuda.synchronize()
    lens, tables = (t.clone() for t in sets[0])
    outs = []
    for i in range(9):
        outs.append(attend(lens, tables))
        lens.fill_(2_000_000_000)
        tables.fill_(-5 if i % 2 else 2_000_000_000)
        lens.copy_(sets[(i + 1) % 3][0])
        tables.copy_(sets[(i + 1) % 3][1])
    for i, out in enumerate(outs):
        assert torch.equal(out, alone[i % 3])
