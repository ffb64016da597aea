"""State rows copied by index through the bulk-copy ring, where its deal of chunks to CTAs can go wrong: one chunk and less,
chunks that end inside a row, more pairs than CTAs, a shared source, a bad index between good ones.  A copy is exact."""

import pytest
import torch

from nano_vllm_jax_b200.kernels import paged_kv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs,conv_bytes,rec_bytes,shared", [
    (1, 16, 16, False), (3, 16384, 16400, False), (24, 48, 65536 + 16, True), (4, 3 * 16384, 9 * 16384 - 16, True),
    (149, 16384 + 32, 112, False), (700, 16, 32, True), (450, 0, 20000, False)])
def test_rows_by_index(pairs, conv_bytes, rec_bytes, shared):
    g = torch.Generator(device="cuda").manual_seed(pairs)
    rows = pairs + 2

    def table(nbytes, dtype):
        if nbytes == 0:
            return None
        return torch.randint(-2 ** 15, 2 ** 15, (rows, nbytes // 2), dtype=torch.int16, device="cuda", generator=g).view(dtype)

    conv_table, conv_pool = table(conv_bytes, torch.bfloat16), table(conv_bytes, torch.bfloat16)
    rec_table, rec_pool = table(rec_bytes, torch.float32), table(rec_bytes, torch.float32)
    src = torch.zeros(pairs, dtype=torch.int64, device="cuda") if shared else torch.randperm(rows, device="cuda", generator=g)[:pairs]
    dst = torch.randperm(rows, device="cuda", generator=g)[:pairs]
    for restore in (False, True):
        want = []
        for t, p in ((conv_table, conv_pool), (rec_table, rec_pool)):
            if t is not None:
                a, b = (p, t) if restore else (t, p)
                w = b.clone().view(torch.int16)
                w[dst] = a.view(torch.int16)[src]
                want.append((b, w))
        ids = (dst, src) if restore else (src, dst)
        if pairs <= paged_kv.HYBRID_HOST_SLOTS:
            ids = tuple(x.tolist() for x in ids)
        else:
            ids = tuple(x.int() for x in ids)
        paged_kv.hybrid_copy(conv_table, rec_table, conv_pool, rec_pool, *ids, restore=restore)
        for b, w in want:
            assert torch.equal(b.view(torch.int16), w)


def test_a_bad_index_leaves_the_other_rows_right():
    t, p = torch.randn(6, 8, 1024, device="cuda"), torch.zeros(6, 8, 1024, device="cuda")
    src = torch.tensor([0, 77, 2, 3], dtype=torch.int32, device="cuda")
    dst = torch.tensor([5, 1, -1, 4], dtype=torch.int32, device="cuda")
    with pytest.raises(paged_kv.DeviceStatusError):
        paged_kv.hybrid_copy(None, t, None, p, src, dst, restore=False)
        paged_kv.check_device_status()
    want = torch.zeros_like(p)
    want[5], want[4] = t[0], t[3]
    assert torch.equal(p, want)


def test_copies_that_follow_one_another_see_each_other():
    """Every copy reads what the one in front of it in the stream has written, with nothing in between to wait for."""
    g = torch.Generator(device="cuda").manual_seed(7)
    table, pool = torch.randn(4, 40_000, device="cuda", generator=g), torch.zeros(4, 40_000, device="cuda")
    k = torch.randn(2, 12, 16, 2, 256, device="cuda", generator=g).bfloat16()
    v = torch.randn(2, 12, 16, 2, 256, device="cuda", generator=g).bfloat16()
    first, k0, v0 = table[0].clone(), k[:, 0].clone(), v[:, 0].clone()
    pairs = [torch.tensor([[i], [i + 1]], dtype=torch.int32, device="cuda") for i in range(11)]
    for i in range(11):  # row 0 -> pool row 0 -> table row 1 -> ..., block 0 -> block 1 -> ...
        paged_kv.hybrid_copy(None, table, None, pool, [i % 4], [i % 4], restore=False)
        paged_kv.hybrid_copy(None, table, None, pool, [(i + 1) % 4], [i % 4], restore=True)
        paged_kv.copy_blocks(k, v, *pairs[i])
    assert all(torch.equal(x, first) for x in (*table, *pool))
    assert all(torch.equal(k[:, i], k0) and torch.equal(v[:, i], v0) for i in range(12))
