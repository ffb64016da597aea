"""Mixed batches (decode rows beside query tiles) through the C ABI and the backend: what the caller lends, how many rows there
are, and calls that follow one another without the host waiting in between."""

import numpy as np
import pytest
import torch

from helpers import BS, SCALE, to_torch

pytestmark = pytest.mark.gpu


def _batch(qlens, cached, seed, layers=1, spare=8):
    """A packed batch whose row r has qlens[r] tokens behind cached[r] cached ones, and N(0, 1) operands for it."""
    rng = np.random.default_rng(seed)
    lens = np.array([q + c for q, c in zip(qlens, cached)], np.int32)
    need = -(-lens // BS)
    pool = int(need.sum()) + spare
    tables, o, perm = np.zeros((len(qlens), int(need.max())), np.int32), 0, rng.permutation(pool)
    for r, n in enumerate(need):
        tables[r, :n] = perm[o:o + n]
        o += n
    pos = np.concatenate([np.arange(c, c + q) for q, c in zip(qlens, cached)]).astype(np.int32)[None]
    rid = np.repeat(np.arange(len(qlens)), qlens).astype(np.int32)[None]
    g = torch.Generator(device="cuda").manual_seed(seed)
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    t = pos.shape[1]
    return {"q": normal(1, t, 8, 256), "k": normal(1, t, 2, 256), "v": normal(1, t, 2, 256),
            "cache": [normal(layers, pool, BS, 2, 256) for _ in range(2)], "tables": to_torch(tables), "lens": to_torch(lens),
            "pos": to_torch(pos), "rid": to_torch(rid), "qsl": to_torch(np.cumsum([0] + list(qlens)).astype(np.int32)),
            "qlens": tuple(qlens)}


def _packed(b, out, status, workspace, nbytes):
    from nano_vllm_jax_b200 import _lib
    k, v = b["cache"]
    return _lib.load().nvj_paged_prefill_packed(
        b["q"].data_ptr(), _lib.NVJ_BF16, k.data_ptr(), v.data_ptr(), _lib.NVJ_BF16, k.shape[1], BS, 2, 256, 8, b["tables"].data_ptr(),
        b["tables"].shape[1], b["lens"].data_ptr(), b["pos"].data_ptr(), b["qsl"].data_ptr(), b["tables"].shape[0], b["q"].shape[1], SCALE,
        out.data_ptr(), status.data_ptr(), workspace, nbytes, 0, torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("nbytes,shift", [(512, 0), (1 << 24, 8)])  # too small; not on a 16-byte boundary
def test_a_workspace_that_cannot_be_used_leaves_the_decode_rows_to_the_tiles(nbytes, shift):
    b = _batch((1, 40, 1, 1, 70), (60, 0, 17, 300, 5), 1)
    out, ref = (torch.full((112 + 1, 2048), float("nan"), device="cuda")[: sum(b["qlens"])] for _ in range(2))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    room = torch.zeros(nbytes + 16, dtype=torch.uint8, device="cuda")
    assert _packed(b, ref, status, None, 0) == 0
    assert _packed(b, out, status, room.data_ptr() + shift, nbytes) == 0
    assert int(status) == 0 and torch.equal(out, ref) and not torch.isnan(out).any() and not room.any()


@pytest.mark.parametrize("chunk", [0, 70])  # decode rows alone, and beside tiles
def test_more_rows_than_a_grid_holds_are_served(chunk):
    rows = 65536 + 3
    qlens = [1] * rows + [chunk] * (chunk > 0)
    n, t = len(qlens), sum(qlens)
    g = torch.Generator(device="cuda").manual_seed(2)
    pool = 64
    cache = [torch.randn((1, pool, BS, 2, 256), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    width = -(-max(chunk, 1) // BS)
    tables = torch.randint(0, pool, (n, width), generator=g, device="cuda", dtype=torch.int32)
    lens = torch.randint(1, BS + 1, (n,), generator=g, device="cuda", dtype=torch.int32)
    q = torch.randn((1, t, 8, 256), generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.full((1, t), width * BS - 1, dtype=torch.int32, device="cuda")
    if chunk:
        lens[-1] = chunk
        pos[0, rows:] = torch.arange(chunk, device="cuda", dtype=torch.int32)
    qsl = to_torch(np.cumsum([0] + qlens).astype(np.int32))
    from nano_vllm_jax_b200.kernels import paged_kv as K
    out = K.packed_paged_prefill_attention(q, cache[0][0], cache[1][0], tables, lens, pos, qsl, BS, SCALE, 4)[0]
    # one block per decode row, in plain torch, the rows behind the grid's limit and some in front of it
    for r in list(range(rows - 5, rows)) + [0, 40000]:
        keys, vals = (c[0, int(tables[r, 0]), : int(lens[r])].float() for c in cache)
        s = torch.einsum("hgd,thd->hgt", q[0, r].float().view(2, 4, 256), keys) * SCALE
        ref = torch.einsum("hgt,thd->hgd", torch.softmax(s, -1), vals).reshape(-1)
        assert float((out[r] - ref).abs().max()) <= 2e-3
    assert not torch.isnan(out).any()


# ---- calls in flight: kernels of one stream overlap (programmatic dependent launch), so nothing may depend on the host waiting

def _calls(kind, n):
    """n calls of one kind, each a function () -> outputs; all of them rewrite the same new rows of the same cache layer, so that
    a call that runs ahead of the one in front, or lags behind it, reads other keys."""
    from nano_vllm_jax_b200.backends import B200Backend
    from nano_vllm_jax_b200.kernels import paged_kv as K
    from nano_vllm_jax_b200.kv_cache import KVCacheStorage
    be = B200Backend()
    g = torch.Generator(device="cuda").manual_seed(9)
    if kind in ("mixed", "mixed, tiles everywhere", "chunk"):
        qlens = {"mixed": (1,) * 32 + (250, 260), "mixed, tiles everywhere": (1,) * 30 + (300,) * 8, "chunk": (40, 130, 342)}[kind]
        b = _batch(qlens, [(37 * i) % 900 + 16 for i in range(len(qlens))], 3)
        md = be.build_attention_metadata(b["pos"], b["tables"], b["lens"], BS, True, query_start_loc=b["qsl"], token_row_ids=b["rid"],
                                         query_lens_host=b["qlens"])
        shape, prefill = (1, sum(qlens)), True
    else:
        rows, width = {"verify 5": (24, 5), "verify 3": (5, 3), "norm": (48, 1), "decode": (16, 1)}[kind]
        b = _batch((width,) * rows, [(53 * i) % 1200 + 3 for i in range(rows)], 4)
        pos = b["pos"].view(rows, width)
        md = be.build_attention_metadata(pos, b["tables"], b["lens"], BS, False,
                                         query_start_loc=None if width == 1 else torch.arange(rows + 1, device="cuda", dtype=torch.int32) * width)
        shape, prefill = (rows, width), False
    cache = KVCacheStorage(*b["cache"])
    normal = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    weight = [normal(256) * 0.1 for _ in range(2)]

    def call(q, k, v):
        if kind == "norm":
            q, _, _ = K.qk_norm_rope_kv_append(q, k, v, *weight, pos, md.slot_mapping, cache.k_cache[0], cache.v_cache[0], eps=1e-6,
                                               rope_theta=1e7, rotary_dim=64)
            return be.attention(0, q, cache, md, BS, SCALE, 4, False)
        return be.write_kv_and_attention(0, q, k, v, cache, md, BS, SCALE, 4, prefill)[1]

    operands = [(normal(*shape, 8, 256), normal(*shape, 2, 256), normal(*shape, 2, 256)) for _ in range(n)]
    return [lambda o=o: call(*o) for o in operands], cache


@pytest.mark.parametrize("kind", ["mixed", "mixed, tiles everywhere", "chunk", "verify 5", "verify 3", "norm", "decode"])
def test_calls_in_flight_give_what_they_give_one_by_one(kind, monkeypatch):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    monkeypatch.setenv("NVJ_CHECK_STATUS", "0")   # no status word read back,
    monkeypatch.setenv("NVJ_POISON_OUTPUT", "0")  # and no fill between two calls
    calls, cache = _calls(kind, 8)
    start = cache.k_cache.clone(), cache.v_cache.clone()
    one_by_one = []
    for c in calls:
        one_by_one.append(c())
        torch.cuda.synchronize()
    after = cache.k_cache.clone(), cache.v_cache.clone()
    for _ in range(20):
        cache.k_cache.copy_(start[0])
        cache.v_cache.copy_(start[1])
        outs = [c() for c in calls]
        for a, b in zip(outs, one_by_one):
            assert torch.equal(a, b)
        assert torch.equal(cache.k_cache, after[0]) and torch.equal(cache.v_cache, after[1])
    K.check_device_status()
    ws = K._workspaces[torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream]
    assert not ws.buf[:64].any()  # the word that lets the decode rows run beside the tiles is left zero


def test_decode_rows_beside_tiles_replay_from_a_graph(monkeypatch):
    from nano_vllm_jax_b200.kernels import paged_kv as K
    monkeypatch.setenv("NVJ_CHECK_STATUS", "0")
    monkeypatch.setenv("NVJ_POISON_OUTPUT", "0")
    monkeypatch.setenv("NVJ_MIXED_SIDE_BY_SIDE", "0")  # one stream, as launched eagerly
    calls, cache = _calls("mixed", 3)
    start = cache.k_cache.clone(), cache.v_cache.clone()
    ref = [c() for c in calls]
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        calls[0]()
    stream.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        outs = [c() for c in calls]
    for _ in range(5):
        cache.k_cache.copy_(start[0])
        cache.v_cache.copy_(start[1])
        graph.replay()
        for a, b in zip(outs, ref):
            assert torch.equal(a, b)
    ws = K._workspaces[torch.cuda.current_device(), stream.cuda_stream]
    torch.cuda.synchronize()
    assert not ws.buf[:64].any()
