"""The staging kernel: sizes around its 16-byte pieces, its CTAs and its grid, and what it leaves to the copy engines."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(dst, src):
    from nano_vllm_jax_b200 import _lib
    n = len(dst)
    pointers = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() for t in ts])  # noqa: E731
    sizes = (ctypes.c_size_t * n)(*[t.numel() * t.element_size() for t in dst])
    return _lib.load().nvj_stage_in(pointers(dst), pointers(src), sizes, n, torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("words", [(1,), (3, 4, 5), (0, 7), (4096, 1, 4095, 4097), (4096 * 64 + 1, 2), (300000, 5, 64, 0, 9, 1, 2, 3)])
def test_sources_arrive_whole_and_nothing_else_is_written(words):
    src = [torch.randint(-1 << 31, (1 << 31) - 1, (w,), dtype=torch.int32).pin_memory() for w in words]
    room = [torch.full((w + 8,), -7, dtype=torch.int32, device="cuda") for w in words]
    for _ in range(2):  # the host writes the same buffers again
        assert _call([r[:w] for r, w in zip(room, words)], src) == 0
        torch.cuda.synchronize()
        for r, s, w in zip(room, src, words):
            assert torch.equal(r[:w].cpu(), s) and bool((r[w:] == -7).all())
            s += 1


def test_other_operands_are_left_alone():
    from nano_vllm_jax_b200 import _lib
    a = torch.zeros(64, dtype=torch.int32, device="cuda")
    pinned = torch.ones(64, dtype=torch.int32).pin_memory()
    for dst, src in (([a], [torch.ones(64, dtype=torch.int32)]), ([a[1:33]], [pinned[:32]]), ([a[:32]], [pinned[1:33]]),
                     ([a] * 9, [pinned] * 9)):
        assert _call(dst, src) == _lib.NVJ_ERR_UNSUPPORTED
    torch.cuda.synchronize()
    assert not a.any()
