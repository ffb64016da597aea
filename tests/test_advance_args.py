"""The lengths and positions that a decode step advances in place: a strided view, whose contiguous copy would be advanced instead
of it, is refused by every entry point that advances."""

import numpy as np
import pytest
import torch

from nano_vllm_jax_b200.kernels import paged_kv as K

ROWS = 6
COLUMN = lambda device: torch.zeros((ROWS, 3), dtype=torch.int32, device=device)  # noqa: E731


@pytest.mark.parametrize("which", ["seq_lens", "positions"])
def test_a_strided_view_is_refused(monkeypatch, which):
    monkeypatch.setattr(K, "_cuda", lambda name, t: t)
    lens, pos = torch.ones(ROWS, dtype=torch.int32), torch.zeros((ROWS, 1), dtype=torch.int32)
    assert K._advance_args((lens, pos, 2, 16), ROWS)[0].data_ptr() == lens.data_ptr()
    lens, pos = (COLUMN("cpu")[:, 1], pos) if which == "seq_lens" else (lens, COLUMN("cpu")[:, 1:2])
    with pytest.raises(ValueError, match="contiguous"):
        K._advance_args((lens, pos, 2, 16), ROWS)


@pytest.mark.parametrize("lens,pos", [(torch.ones(ROWS), None), (torch.ones(ROWS, dtype=torch.int32), torch.ones(ROWS)),
                                      (torch.ones(ROWS - 1, dtype=torch.int32), None)])
def test_other_types_and_sizes_are_refused_as_before(monkeypatch, lens, pos):
    monkeypatch.setattr(K, "_cuda", lambda name, t: t)
    with pytest.raises(ValueError):
        K._advance_args((lens, pos, 2, 16), ROWS)


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["seq_lens", "positions"])
def test_the_entry_points_refuse_it_before_they_launch(which):
    from helpers import BS, SCALE, decode_case, to_torch
    c = decode_case(3, 64, ROWS, 1, 1, width=2)
    q, nk, nv, k, v = (to_torch(c[n]) for n in ("q", "new_k", "new_v", "k_cache", "v_cache"))
    tables = to_torch(np.arange(2 * ROWS, dtype=np.int32).reshape(ROWS, 2))
    lens, pos = torch.full((ROWS,), 5, dtype=torch.int32, device="cuda"), torch.zeros((ROWS, 1), dtype=torch.int32, device="cuda")
    tokens, k0 = torch.zeros(ROWS, dtype=torch.int32, device="cuda"), k.clone()
    if which == "seq_lens":
        lens = (COLUMN("cuda") + 5)[:, 1]
    else:
        pos = COLUMN("cuda")[:, 1:2]
    with pytest.raises(ValueError, match="contiguous"):
        K.paged_decode_step(q, nk, nv, k, v, tables, lens, pos, 0, BS, SCALE, 4, tokens)
    with pytest.raises(ValueError, match="contiguous"):
        K.row_argmax(torch.randn((ROWS, 64), device="cuda"), advance=(lens, pos, 2, BS))
    assert torch.equal(k, k0) and lens.tolist() == [5] * ROWS
