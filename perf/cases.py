"""Workloads of the paged KV-cache path as a serving program runs them, for timing and for comparing outputs.

Every case goes through the package's public entry points with the model's head layout (8 query heads over 2 KV heads,
head_dim 256, 16-token blocks, scale 1/16) and N(0, 1) values, over blocks scattered in the pool.  `prepare` makes what a
program holds before the call, `run` is one pass, `work` the bytes and operations that the pass cannot do without.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

from nano_vllm_jax_b200.backends import B200Backend
from nano_vllm_jax_b200.engine.block_manager import BlockManager
from nano_vllm_jax_b200.engine.prefix_state import HybridStateTable, PrefixStateCache
from nano_vllm_jax_b200.engine.resident_decode import DecodeStepGraph, ResidentDecodeMetadata
from nano_vllm_jax_b200.engine.scheduled_batch import build_mixed_prefill_decode_batch
from nano_vllm_jax_b200.engine.sequence import Sequence
from nano_vllm_jax_b200.host_pipeline import HostDecodePipeline
from nano_vllm_jax_b200.kernels import paged_kv
from nano_vllm_jax_b200.kv_cache import KVCacheSpec, KVCacheStorage

BS, HQ, HKV, D, GROUPS = 16, 8, 2, 256, 4
SCALE = D ** -0.5
ROTARY, THETA, EPS = 64, 1e7, 1e-6
GDN_CONV, GDN_REC = (18, 6144, 4), (18, 16, 128, 128)  # one sequence's GDN state: 18 layers, bf16 and fp32
DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}
MOST_TOKENS = 128 * 20480  # live tokens of the largest case: 5.4 GB of K and V


# ------------------------------------------------------------------------------------------------ the cases

def listed():
    return [
        # one attention layer of a decode step for a handful of short requests: latency is all there is
        {"name": "decode_4_rows", "kind": "decode", "rows": 4, "lo": 64, "hi": 512, "dtype": "bfloat16"},
        # few long conversations: one row has far more keys than one SM should walk
        {"name": "decode_8_long_rows", "kind": "decode", "rows": 8, "lo": 8192, "hi": 32768, "dtype": "bfloat16"},
        # one GPU's share of a large long-context deployment: the largest decode batch
        {"name": "decode_128_long_rows", "kind": "decode", "rows": 128, "lo": 8192, "hi": 32768, "dtype": "bfloat16"},
        # the cache-dtype override to fp32 (the format of the reference project's own CUDA routes and their 8-row workload)
        {"name": "decode_8_rows_fp32", "kind": "decode", "rows": 8, "lo": 64, "hi": 512, "dtype": "float32"},
        # decode-heavy serving: a full batch installed once and stepped from a CUDA graph over resident metadata
        {"name": "graph_256_rows", "kind": "graph", "rows": 256, "lo": 1024, "hi": 4096, "steps": 8},
        # the same from host memory: operands copied in and results copied out on every step
        {"name": "host_64_rows", "kind": "host", "rows": 64, "lo": 512, "hi": 4096, "steps": 8},
        # verification of speculated tokens: five query tokens per row, appended and attended in one call
        {"name": "verify_64x5", "kind": "verify", "rows": 64, "width": 5, "lo": 1024, "hi": 4096},
        # chunked prefill: a 512-token chunk made up of three requests at different depths
        {"name": "prefill_chunk_512", "kind": "prefill", "rows": 3, "tokens": 512, "cached": 1024, "pad": 0},
        # a long prompt in one chunk: the largest prefill
        {"name": "prefill_16384", "kind": "prefill", "rows": 1, "tokens": 16384, "cached": 0, "pad": 0},
        # continuous batching: 32 decode rows and two 256-token chunks through six layers, from the scheduler's sequences
        {"name": "mixed_step_6_layers", "kind": "mixed", "rows": 32, "lo": 128, "hi": 2048, "chunks": 2, "chunk": 256, "layers": 6},
        # a model's decode step over its six full-attention layers: norm + RoPE + append, then attention
        {"name": "layers_48_rows", "kind": "layers", "rows": 48, "lo": 128, "hi": 2048, "layers": 6},
        # four requests that share a cached 512-token prefix are admitted: blocks, GDN state, a private copy of the prefix
        {"name": "prefix_hit_4", "kind": "prefix", "requests": 4, "prefix": 512, "prompt": 1536, "layers": 6},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _contexts(rng, case, hi_lo, hi_hi):
    """Context range of a drawn batch, and as many rows as the largest case has room for."""
    case["hi"] = _log(rng, hi_lo, hi_hi)
    case["lo"] = max(16, case["hi"] // rng.choice((2, 4, 8)))
    case["rows"] = max(1, min(case["rows"], MOST_TOKENS * 2 // (case["lo"] + case["hi"])))
    return case


def draw(rng):
    kind = rng.choice(("decode", "decode", "decode", "graph", "host", "verify", "prefill", "prefill", "mixed", "layers", "prefix"))
    if kind == "decode":
        dtype = rng.choice(("bfloat16", "bfloat16", "bfloat16", "float32", "float16"))
        if dtype == "bfloat16":
            return _contexts(rng, {"kind": kind, "rows": _log(rng, 1, 256), "dtype": dtype}, 64, 32768)
        return _contexts(rng, {"kind": kind, "rows": _log(rng, 1, 32), "dtype": dtype}, 64, 2048)
    if kind == "graph":
        return _contexts(rng, {"kind": kind, "rows": _log(rng, 1, 256), "steps": 8}, 128, 4096)
    if kind == "host":
        return _contexts(rng, {"kind": kind, "rows": _log(rng, 4, 256), "steps": 8}, 128, 4096)
    if kind == "verify":
        return _contexts(rng, {"kind": kind, "rows": _log(rng, 1, 256), "width": rng.randint(2, 9)}, 128, 4096)
    if kind == "prefill":
        tokens = _log(rng, 17, 12000)
        return {"kind": kind, "rows": max(1, min(rng.randint(1, 8), tokens // 16)), "tokens": tokens,
                "cached": rng.choice((0, _log(rng, 16, 4096))), "pad": rng.choice((0, -tokens % 64))}
    if kind == "mixed":
        case = _contexts(rng, {"kind": kind, "rows": _log(rng, 2, 96)}, 128, 2048)
        return dict(case, chunks=rng.randint(1, 4), chunk=_log(rng, 24, 512), layers=6)
    if kind == "layers":
        return dict(_contexts(rng, {"kind": kind, "rows": _log(rng, 1, 256)}, 64, 4096), layers=6)
    prefix = 16 * _log(rng, 4, 64)
    return {"kind": kind, "requests": rng.randint(1, 12), "prefix": prefix, "prompt": prefix + _log(rng, 33, 1500), "layers": 6}


# ------------------------------------------------------------------------------------------------ sizes

def _spread(lo, hi, n):
    """n lengths over [lo, hi], evenly."""
    return [int(round(lo + (hi - lo) * (i + 0.5) / n)) for i in range(n)]


def _chunks(case):
    """(chunk length, tokens already cached) of a prefill batch's rows: ragged, every row at another depth."""
    n, tokens = case["rows"], case["tokens"]
    cuts = [tokens * i * (i + 1) // (n * (n + 1)) for i in range(n + 1)]
    return [(cuts[i + 1] - cuts[i], case["cached"] * (n - i) // n) for i in range(n)]


def _mixed_rows(case):
    """Row lengths of a mixed step: decode rows' contexts (this step's token counted), then (chunk, cached) of the chunks."""
    return _spread(case["lo"], case["hi"], case["rows"]), [(case["chunk"], case["chunk"] * (i % 2)) for i in range(case["chunks"])]


def work(case):
    """Every live K and V row, query, table entry and new row read once, every output and new row written once."""
    kind, item = case["kind"], DTYPES[case.get("dtype", "bfloat16")].itemsize
    token = 2 * HKV * D * item  # one token's K and V

    def decode(lens, width=1):
        n = len(lens) * width
        return (sum(lens) * token + n * token * 2 + n * HQ * D * (item + 4) + sum(-(-x // BS) for x in lens) * 4 + n * 12,
                4 * HQ * D * sum(lens) * width)

    def prefill(rows):
        tokens, live = sum(c for c, _ in rows), sum(c + p for c, p in rows)
        return (live * token + tokens * token * 2 + tokens * (HQ * D * 6 + 12) + live // BS * 4,
                4 * HQ * D * sum(c * p + c * (c + 1) // 2 for c, p in rows))

    if kind in ("decode", "verify"):
        nbytes, flops = decode(_spread(case["lo"], case["hi"], case["rows"]), case.get("width", 1))
    elif kind in ("graph", "host"):
        nbytes, flops = 0, 0
        for s in range(case["steps"]):
            b, f = decode([x + s for x in _spread(case["lo"], case["hi"], case["rows"])])
            nbytes, flops = nbytes + b, flops + f
    elif kind == "prefill":
        nbytes, flops = prefill(_chunks(case))
    elif kind == "mixed":
        lens, chunks = _mixed_rows(case)
        (b0, f0), (b1, f1) = decode(lens), prefill(chunks)
        nbytes, flops = case["layers"] * (b0 + b1), case["layers"] * (f0 + f1)
    elif kind == "layers":
        b, f = decode(_spread(case["lo"], case["hi"], case["rows"]))
        n = case["rows"]
        nbytes, flops = case["layers"] * (b + n * HQ * D * 4), case["layers"] * f
    else:
        state = math.prod(GDN_CONV) * 2 + math.prod(GDN_REC) * 4
        n, prefix = case["requests"], case["prefix"] * case["layers"] * token
        nbytes, flops = (n + 1) * prefix + (3 * n + 1) * state, 0  # one stored prefix and state serve all n; n snapshots
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "prefix":
        return "exact"  # copies
    if case.get("dtype") == "float32":
        return {"rel": 1e-5, "max": 2e-4}
    if case.get("dtype") == "float16":
        return {"rel": 5e-4, "max": 5e-3}
    return {"rel": 3e-3, "max": 3e-2}  # bf16 operands: softmax weights within a bf16 rounding, fp32 sums


# ------------------------------------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, dtype, *shape):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=g)


def _cache(g, layers, blocks, dtype=torch.bfloat16):
    storage = B200Backend().allocate_kv_cache(KVCacheSpec(layers, blocks, BS, HKV, D, dtype), 1, 1)
    storage.k_cache.normal_(generator=g)
    storage.v_cache.normal_(generator=g)
    return storage


def _tables(g, room):
    """Block tables for rows that need room for `room[b]` tokens, over a pool a quarter larger than that; unused entries 0."""
    need = [-(-r // BS) for r in room]
    pool = sum(need) + sum(need) // 4 + 8
    ids = torch.randperm(pool, generator=g, device="cuda").to(torch.int32)
    mask = torch.arange(max(need), device="cuda")[None] < torch.tensor(need, device="cuda")[:, None]
    tables = torch.zeros(len(need), max(need), dtype=torch.int32, device="cuda")
    tables[mask] = ids[: sum(need)]
    return tables, pool


def _int(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _lengths(case, seed):
    lens = _spread(case["lo"], case["hi"], case["rows"])
    random.Random(seed).shuffle(lens)
    return lens


def _fragmented(num_blocks, seed):
    """A block manager whose free list is in the order that a server leaves it in after many requests: shuffled."""
    manager = BlockManager(num_blocks, BS)
    gone = [Sequence([0] * (BS * min(8, num_blocks - i)), seq_id=i) for i in range(0, num_blocks, 8)]
    for s in gone:
        manager.allocate(s, use_prefix_cache=False)
    random.Random(seed).shuffle(gone)
    for s in gone:
        manager.deallocate(s)
    return manager


def _prepare_decode(case, seed):
    g, dtype = _gen(seed), DTYPES[case["dtype"]]
    lens = _lengths(case, seed)
    tables, pool = _tables(g, lens)
    n = case["rows"]
    return {"backend": B200Backend(), "cache": _cache(g, 1, pool, dtype), "tables": tables, "lens": _int(lens),
            "pos": _int([[x - 1] for x in lens]), "q": _normal(g, dtype, n, 1, HQ, D),
            "k": _normal(g, dtype, n, 1, HKV, D), "v": _normal(g, dtype, n, 1, HKV, D)}


def _run_decode(s):
    md = s["backend"].build_attention_metadata(s["pos"], s["tables"], s["lens"], BS, False)
    cache, out = s["backend"].write_kv_and_attention(0, s["q"], s["k"], s["v"], s["cache"], md, BS, SCALE, GROUPS, False)
    return out, cache.k_cache, cache.v_cache


def _prepare_graph(case, seed):
    g, n = _gen(seed), case["rows"]
    before = [x - 1 for x in _lengths(case, seed)]  # lengths before the first step's token
    tables, pool = _tables(g, [x + case["steps"] + 1 for x in before])
    cache = _cache(g, 1, pool)
    meta = ResidentDecodeMetadata(n, tables.shape[1], BS)
    host = (tables.cpu().numpy(), np.array(before, np.int32))
    meta.load(*host)
    graph = DecodeStepGraph(meta, cache.k_cache, cache.v_cache, 0, SCALE, GROUPS)
    for t in (graph.query, graph.new_k, graph.new_v):
        t.normal_(generator=g)
    graph.capture()
    return {"graph": graph, "meta": meta, "host": host, "steps": case["steps"], "cache": cache}


def _run_graph(s):
    s["meta"].load(*s["host"])
    for _ in range(s["steps"]):
        out, tokens = s["graph"].replay()
    return out, tokens, s["meta"].seq_lens, s["cache"].k_cache, s["cache"].v_cache


def _prepare_host(case, seed):
    g, n = _gen(seed), case["rows"]
    lens = _lengths(case, seed)
    tables, pool = _tables(g, [x + case["steps"] for x in lens])
    cache = _cache(g, 1, pool)

    def pinned(t):
        return t.cpu().pin_memory()

    steps = [(pinned(_normal(g, torch.bfloat16, n, 1, HQ, D)), pinned(_normal(g, torch.bfloat16, n, 1, HKV, D)),
              pinned(_normal(g, torch.bfloat16, n, 1, HKV, D)), pinned(_int([[x - 1 + s] for x in lens])),
              pinned(_int([x + s for x in lens]))) for s in range(case["steps"])]
    pipe = HostDecodePipeline(B200Backend(), cache, n, tables.shape[1], BS, SCALE, GROUPS, depth=2, capture=True)
    return {"pipe": pipe, "steps": steps, "tables": pinned(tables), "cache": cache,
            "outs": torch.empty(case["steps"], n, 1, HQ * D)}


def _run_host(s):
    pipe, outs, last = s["pipe"], s["outs"], None
    for i, (q, k, v, pos, lens) in enumerate(s["steps"]):
        ticket = pipe.submit(0, q, k, v, s["tables"], pos, lens)
        if i > 0:
            outs[i - 1].copy_(pipe.result(last))
        last = ticket
    outs[len(s["steps"]) - 1].copy_(pipe.result(last))
    return outs, s["cache"].k_cache, s["cache"].v_cache


def _prepare_verify(case, seed):
    g, n, w = _gen(seed), case["rows"], case["width"]
    lens = [max(x, w) for x in _lengths(case, seed)]
    tables, pool = _tables(g, lens)
    return {"backend": B200Backend(), "cache": _cache(g, 1, pool), "tables": tables, "lens": _int(lens),
            "pos": _int([[x - w + t for t in range(w)] for x in lens]), "qsl": _int([i * w for i in range(n + 1)]),
            "q": _normal(g, torch.bfloat16, n, w, HQ, D), "k": _normal(g, torch.bfloat16, n, w, HKV, D),
            "v": _normal(g, torch.bfloat16, n, w, HKV, D)}


def _run_verify(s):
    md = s["backend"].build_attention_metadata(s["pos"], s["tables"], s["lens"], BS, False, query_start_loc=s["qsl"])
    cache, out = s["backend"].write_kv_and_attention(0, s["q"], s["k"], s["v"], s["cache"], md, BS, SCALE, GROUPS, False)
    return out, cache.k_cache, cache.v_cache


def _prepare_prefill(case, seed):
    g = _gen(seed)
    rows = _chunks(case)
    random.Random(seed).shuffle(rows)
    tables, pool = _tables(g, [c + p for c, p in rows])
    bucket = case["tokens"] + case["pad"]
    pos = [p + i for c, p in rows for i in range(c)] + [0] * case["pad"]
    rid = [r for r, (c, _) in enumerate(rows) for _ in range(c)] + [0] * case["pad"]
    return {"backend": B200Backend(), "cache": _cache(g, 1, pool), "tables": tables, "lens": _int([c + p for c, p in rows]),
            "pos": _int([pos]), "rid": _int([rid]), "qsl": _int(np.cumsum([0] + [c for c, _ in rows]).tolist()),
            "qlens": tuple(c for c, _ in rows), "q": _normal(g, torch.bfloat16, 1, bucket, HQ, D),
            "k": _normal(g, torch.bfloat16, 1, bucket, HKV, D), "v": _normal(g, torch.bfloat16, 1, bucket, HKV, D)}


def _run_prefill(s):
    md = s["backend"].build_attention_metadata(s["pos"], s["tables"], s["lens"], BS, True, query_start_loc=s["qsl"],
                                               token_row_ids=s["rid"], query_lens_host=s["qlens"])
    cache, out = s["backend"].write_kv_and_attention(0, s["q"], s["k"], s["v"], s["cache"], md, BS, SCALE, GROUPS, True)
    return out, cache.k_cache, cache.v_cache


def _prepare_mixed(case, seed):
    g, r = _gen(seed), random.Random(seed)
    lens, chunks = _mixed_rows(case)
    r.shuffle(lens)
    prompts = [2 * case["chunk"]] * len(chunks)
    manager = _fragmented(sum(-(-x // BS) + 1 for x in lens + prompts) * 5 // 4, seed)
    sequences = [Sequence([r.randrange(1, 150_000) for _ in range(x)], seq_id=i) for i, x in enumerate(lens + prompts)]
    for s in sequences:
        manager.allocate(s, use_prefix_cache=False)
    decode, prefill = sequences[: len(lens)], sequences[len(lens):]
    for s, (_, cached) in zip(prefill, chunks):
        s.num_cached_tokens = cached
    tokens = len(lens) + sum(c for c, _ in chunks)
    layers = [tuple(_normal(g, torch.bfloat16, 1, tokens, h, D) for h in (HQ, HKV, HKV)) for _ in range(case["layers"])]
    return {"backend": B200Backend(), "cache": _cache(g, case["layers"], len(manager.blocks)), "manager": manager,
            "decode": decode, "prefill": prefill, "chunks": [c for c, _ in chunks], "layers": layers}


def _run_mixed(s):
    backend, cache, outs = s["backend"], s["cache"], []
    for seq in s["decode"]:
        s["manager"].may_append_slots(seq, 1)
    b = build_mixed_prefill_decode_batch(decode_seqs=s["decode"], prefill_seqs=s["prefill"], prefill_chunk_lens=s["chunks"])
    md = backend.build_attention_metadata(b.positions, b.block_tables, b.seq_lens, BS, True, query_start_loc=b.query_start_loc,
                                          num_prefill_tokens=b.num_prefill_tokens, num_decode_tokens=b.num_decode_tokens,
                                          token_row_ids=b.token_row_ids, query_lens_host=b.query_lens_host)
    for i, (q, k, v) in enumerate(s["layers"]):
        cache, out = backend.write_kv_and_attention(i, q, k, v, cache, md, BS, SCALE, GROUPS, True)
        outs.append(out)
    return outs, cache.k_cache, cache.v_cache


def _prepare_layers(case, seed):
    g, n = _gen(seed), case["rows"]
    lens = _lengths(case, seed)
    tables, pool = _tables(g, lens)
    layers = [{"qg": _normal(g, torch.bfloat16, n, 1, HQ, 2 * D), "k": _normal(g, torch.bfloat16, n, 1, HKV, D),
               "v": _normal(g, torch.bfloat16, n, 1, HKV, D), "qw": _normal(g, torch.bfloat16, D) * 0.1,
               "kw": _normal(g, torch.bfloat16, D) * 0.1} for _ in range(case["layers"])]
    return {"backend": B200Backend(), "cache": _cache(g, case["layers"], pool), "tables": tables, "lens": _int(lens),
            "pos": _int([[x - 1] for x in lens]), "layers": layers}


def _run_layers(s):
    backend, cache, outs = s["backend"], s["cache"], []
    md = backend.build_attention_metadata(s["pos"], s["tables"], s["lens"], BS, False)
    for i, w in enumerate(s["layers"]):
        # the query is the first half of the query|gate projection
        q, _, _ = paged_kv.qk_norm_rope_kv_append(w["qg"][..., :D], w["k"], w["v"], w["qw"], w["kw"], s["pos"], md.slot_mapping,
                                                  cache.k_cache[i], cache.v_cache[i], eps=EPS, rope_theta=THETA, rotary_dim=ROTARY)
        outs.append(backend.attention(i, q, cache, md, BS, SCALE, GROUPS, False))
    return outs, cache.k_cache, cache.v_cache


def _prepare_prefix(case, seed):
    g, r, n = _gen(seed), random.Random(seed), case["requests"]
    shared = [r.randrange(1, 150_000) for _ in range(case["prefix"])]
    prefix_blocks = case["prefix"] // BS
    blocks = prefix_blocks + n * -(-case["prompt"] // BS) + 64
    manager = _fragmented(blocks, seed)
    cache = _cache(g, case["layers"], blocks + n * prefix_blocks)  # the private copies lie behind the managed pool
    table = HybridStateTable(GDN_CONV, GDN_REC, max_slots=n + 1, conv_dtype=torch.bfloat16)
    states = PrefixStateCache(table, capacity=n + 2)
    donor = Sequence(shared, seq_id=n)
    manager.allocate(donor, cacheable_hashes=states.cacheable_hashes)
    state = table.state(n)
    state.conv_state.normal_(generator=g)
    state.recurrent_state.normal_(generator=g)
    table.mark_written([n])
    states.record_computed_prefix_states(manager, [donor], [len(shared)])
    requests = [Sequence(shared + [r.randrange(1, 150_000) for _ in range(case["prompt"] - case["prefix"])], seq_id=i) for i in range(n)]
    src = _int(list(donor.block_table) * n)
    dst = torch.arange(blocks, blocks + n * prefix_blocks, dtype=torch.int32, device="cuda")
    return {"manager": manager, "cache": cache, "table": table, "states": states, "requests": requests, "src": src, "dst": dst,
            "own": [r.getrandbits(62) for _ in range(n)], "prefix": case["prefix"]}


def _run_prefix(s):
    manager, states, requests = s["manager"], s["states"], s["requests"]
    for seq in requests:
        if not manager.can_allocate(seq, cacheable_hashes=states.cacheable_hashes):
            raise RuntimeError("no room for the request")
        manager.allocate(seq, cacheable_hashes=states.cacheable_hashes)
    cached = [seq.num_cached_tokens for seq in requests]
    states.pin_for(requests)
    states.install_cached_prefix_hybrid_states(requests)
    paged_kv.copy_blocks(s["cache"].k_cache, s["cache"].v_cache, s["src"], s["dst"])
    states.snapshot([seq.seq_id for seq in requests], s["own"])
    for seq in requests:
        manager.deallocate(seq)
    return (cached, s["table"].conv, s["table"].rec, states.conv_pool, states.rec_pool, s["cache"].k_cache, s["cache"].v_cache)


_PREPARE = {"decode": _prepare_decode, "graph": _prepare_graph, "host": _prepare_host, "verify": _prepare_verify,
            "prefill": _prepare_prefill, "mixed": _prepare_mixed, "layers": _prepare_layers, "prefix": _prepare_prefix}
_RUN = {"decode": _run_decode, "graph": _run_graph, "host": _run_host, "verify": _run_verify, "prefill": _run_prefill,
        "mixed": _run_mixed, "layers": _run_layers, "prefix": _run_prefix}


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return _RUN[state["kind"]](state)
