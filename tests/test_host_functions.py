"""Block bookkeeping and batch layout without the host extension: the modules import, and the Python forms give what the
extension gives."""

import random
import subprocess
import sys
from pathlib import Path

import pytest
import torch

from nano_vllm_jax_b200 import _lib
from nano_vllm_jax_b200.engine import block_manager, host_functions
from nano_vllm_jax_b200.engine.sequence import Sequence

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.parametrize("fault", ["ImportError('libtorch_cuda.so')", "FileNotFoundError('g++')", "RuntimeError('g++ failed')"])
def test_the_engine_modules_import_without_the_extension(fault):
    code = (f"from nano_vllm_jax_b200 import _lib\n"
            f"def missing(): raise {fault}\n"
            f"_lib.host_module = missing\n"
            f"import torch; torch.cuda.is_available = lambda: False\n"
            f"from nano_vllm_jax_b200.engine.block_manager import BlockManager\n"
            f"from nano_vllm_jax_b200.engine.scheduled_batch import build_decode_batch\n"
            f"from nano_vllm_jax_b200.engine.sequence import Sequence\n"
            f"m, s = BlockManager(8, 4), Sequence([1, 2, 3, 4, 5], seq_id=0)\n"
            f"m.allocate(s); b = build_decode_batch([s], device='cpu')\n"
            f"assert s.block_table == [0, 1] and b.block_tables.tolist() == [[0, 1]]\n")
    subprocess.run([sys.executable, "-c", code], check=True, cwd=ROOT)


def test_with_a_gpu_a_missing_extension_is_an_error(monkeypatch):
    def missing():
        raise ImportError("no extension")
    monkeypatch.setattr(_lib, "host_module", missing)
    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    with pytest.raises(ImportError):
        host_functions.load()


def _run(functions, monkeypatch, seed):
    """A random life of a pool under one set of functions; everything that the manager's state shows on the way."""
    monkeypatch.setattr(block_manager, "_host", functions)
    monkeypatch.setattr(block_manager, "_hash_chain", functions.hash_chain)
    r, bs = random.Random(seed), 4
    m, live, seen = block_manager.BlockManager(40, bs), [], []
    prompts = [[r.randrange(50) for _ in range(24)] for _ in range(3)]
    for step in range(200):
        if live and (r.random() < 0.45 or len(live) > 6):
            m.deallocate(live.pop(r.randrange(len(live))))
        else:
            s = Sequence(prompts[r.randrange(3)][: r.randrange(1, 24)] + [r.randrange(50) for _ in range(r.randrange(9))], seq_id=step)
            cacheable = None if r.random() < 0.5 else {m.compute_hash(s.token_ids[:bs])}
            seen.append(m.can_allocate(s, cacheable_hashes=cacheable))
            if seen[-1]:
                m.allocate(s, use_prefix_cache=r.random() < 0.8, cacheable_hashes=cacheable)
                m.record_computed_prefix(s, s.num_tokens, publish=True)
                seen.append((list(s.block_table), s.num_cached_tokens, s.cached_prefix_hash))
                live.append(s)
        seen.append((list(m.free_block_ids), sorted(m.used_block_ids), dict(m.hash_to_block_id),
                     [(b.ref_count, b.hash, list(b.token_ids)) for b in m.blocks]))
    return seen


@pytest.mark.parametrize("seed", range(4))
def test_the_python_forms_manage_blocks_alike(seed, monkeypatch):
    assert _run(_lib.host_module(), monkeypatch, seed) == _run(host_functions, monkeypatch, seed)


@pytest.mark.parametrize("parts,rows,width", [([([1, 2], (2,)), ([3], (2, 2)), ([], (0,))], [[7, 8], [], (9,)], 3), ([], [[]], 0),
                                              ([([2**31 - 1, -(2**31)], (1, 2))], [], 4)])
def test_the_python_form_packs_alike(parts, rows, width):
    a, b = (f.pack_batch(parts, rows, width, -1) for f in (_lib.host_module(), host_functions))
    assert [t.tolist() for t in a[0]] == [t.tolist() for t in b[0]] and a[1].tolist() == b[1].tolist() and a[2] == b[2]
    assert all(x.shape == y.shape and x.dtype == y.dtype == torch.int32 for x, y in zip(a[0] + [a[1]], b[0] + [b[1]]))


@pytest.mark.parametrize("parts,rows,error", [([([1, 2, 3], (2,))], [], ValueError), ([([2**31], (1,))], [], OverflowError),
                                              ([], [[1, 2, 3]], ValueError), ([], [[-(2**31) - 1]], OverflowError)])
def test_the_python_form_refuses_alike(parts, rows, error):
    messages = []
    for f in (_lib.host_module(), host_functions):
        with pytest.raises(error) as e:
            f.pack_batch(parts, rows, 2, -1)
        messages.append(str(e.value))
    assert messages[0] == messages[1]


# no room for the rest behind shared blocks, tokens that are no machine-size integers (equal ones share all the same), a tuple of tokens
@pytest.mark.parametrize("tokens", [list(range(9)) + [7] * 40, [1, 2, 3, 4, 5.0, 6], [0, 1, 2, 3, 2 ** 70, 5, 6, 7], tuple(range(8)), [True, 1, 2, 3, 4]])
def test_an_allocation_in_one_call_leaves_what_the_steps_leave(tokens, monkeypatch):
    def life(functions):
        monkeypatch.setattr(block_manager, "_host", functions)
        monkeypatch.setattr(block_manager, "_hash_chain", functions.hash_chain)
        m = block_manager.BlockManager(8, 4)
        first, gone, s = Sequence(range(8), seq_id=0), Sequence([1] * 12, seq_id=1), Sequence([0], seq_id=2)
        for q in (first, gone):
            m.allocate(q)
            m.record_computed_prefix(q, q.num_tokens, publish=True)
        m.deallocate(gone)
        s.token_ids, s.num_tokens = tokens, len(tokens)
        try:
            m.allocate(s)
            error = None
        except (StopIteration, OverflowError, TypeError) as e:
            error = type(e)
        return (error, s.block_table, s.num_cached_tokens, s.cached_prefix_hash, list(m.free_block_ids), sorted(m.used_block_ids), dict(m.hash_to_block_id),
                [(b.ref_count, b.hash, list(b.token_ids)) for b in m.blocks])

    assert life(_lib.host_module()) == life(host_functions)
