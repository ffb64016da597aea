"""The host extension's chained block digests against the xxhash package, over every remainder of its four-word stripes."""

import numpy as np
import pytest
import xxhash

from nano_vllm_jax_b200.engine.block_manager import BlockManager, _hash_chain


@pytest.mark.parametrize("block_size", [1, 2, 3, 4, 5, 7, 8, 16, 33])
@pytest.mark.parametrize("prefix", [-1, 0, 7, (1 << 64) - 1])
def test_hash_chain_equals_xxh64_over_prefix_and_int64_tokens(block_size, prefix):
    tokens = np.random.default_rng(block_size).integers(-(1 << 62), 1 << 62, size=3 * block_size + block_size // 2).tolist()
    got, h = _hash_chain(tokens, block_size, 3, prefix), prefix
    for i in range(3):
        d = xxhash.xxh64()
        if h != -1:
            d.update(h.to_bytes(8, "little"))
        d.update(np.asarray(tokens[i * block_size:(i + 1) * block_size], np.int64).tobytes())
        h = d.intdigest()
        assert got[i] == h
    assert BlockManager.compute_hash(tokens[:block_size], prefix) == got[0]
    assert _hash_chain([1, 2.0], 2, 1, -1) is None and _hash_chain([1, 1 << 64], 2, 1, -1) is None
