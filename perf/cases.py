"""The workloads whose speed this library answers for, as a host program drives them through `mechta_b200.kv`.

One pass is one call order of a host: a verify step of all attention layers, a fused layer step, a step on the ring caches
of sliding layers, one step of many sessions, a prefill block, or a turn that starts from a stored prefix. `listed()` names
the cases, `draw()` gives others from the same ranges; sizes come from the benchmark's configurations and from the tests,
with odd ones among them.
"""
from __future__ import annotations

import functools
import math

import torch

from mechta_b200 import kv

LAYERS = 10  # full-attention layers of the reference's model
ROW_ELEMS = 2 * kv.ROW  # K and V elements of one position


def listed():
    return [
        # The smallest call: one layer's 4-token verify step at 4,096 tokens (append, attention, rollback).
        {"name": "verify_4k", "kind": "verify", "fmt": "f16", "layers": 1, "tokens": 4096, "ntok": 4},
        # A chat that has just begun, decoded without drafts: every layer's fused step on a short history. Launches count.
        {"name": "step_chat", "kind": "step", "fmt": "f16", "layers": LAYERS, "tokens": 1777, "ntok": 1},
        # Sliding-window layers with attention sinks on a ring cache of 1,024 rows that has gone round many times.
        {"name": "window_ring", "kind": "window", "fmt": "f16", "layers": LAYERS, "tokens": 20011, "ntok": 4, "ring": 1024, "window": 513},
        # The steady-state decode configuration: 10 layers, f16 cache at 65,536 tokens, 4-token verify.
        {"name": "verify_65k", "kind": "verify", "fmt": "f16", "layers": LAYERS, "tokens": 65536, "ntok": 4},
        # A long chat at an odd length with 3 tokens a step, each layer's rows written just before its attention.
        {"name": "step_24k", "kind": "step", "fmt": "f16", "layers": LAYERS, "tokens": 23451, "ntok": 3},
        # The f32 cache (hosts that keep full precision) at an ordinary odd length, one draft a step.
        {"name": "verify_f32_9k", "kind": "verify", "fmt": "f32", "layers": LAYERS, "tokens": 9001, "ntok": 2},
        # The longest context on the f32 cache.
        {"name": "verify_f32_262k", "kind": "verify", "fmt": "f32", "layers": LAYERS, "tokens": 262000, "ntok": 4},
        # A server's step: 32 sessions with ragged lengths, one batched attention launch per layer.
        {"name": "sessions_32", "kind": "sessions", "fmt": "f16", "layers": 4, "sessions": 32, "shortest": 1024, "longest": 131072, "ntok": 4},
        # A 2,048-token block over a 32,768-token prefix, f16 queries.
        {"name": "prefill_2k", "kind": "prefill", "fmt": "f16", "layers": LAYERS, "prefix": 32768, "ntok": 2048, "q": "f16"},
        # A follow-up message of ordinary, ragged size behind a history, f32 queries.
        {"name": "prefill_200", "kind": "prefill", "fmt": "f16", "layers": LAYERS, "prefix": 9001, "ntok": 200, "q": "f32"},
        # The same kind of block on the f32 cache.
        {"name": "prefill_f32", "kind": "prefill", "fmt": "f32", "layers": LAYERS, "prefix": 4096, "ntok": 512, "q": "f32"},
        # A turn of a stored conversation: restore the prefix from pinned memory, prefill the message, snapshot the result.
        {"name": "stored_turn", "kind": "turn", "fmt": "f16", "layers": LAYERS, "prefix": 12345, "ntok": 160, "q": "f32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["verify", "verify", "step", "window", "sessions", "prefill", "prefill", "turn"])
    fmt = rng.choice(["f16", "f16", "f32"])
    layers = rng.randint(1, LAYERS)
    if kind in ("verify", "step"):
        return {"kind": kind, "fmt": fmt, "layers": layers, "tokens": _log(rng, 500, 262000), "ntok": rng.randint(1, 4)}
    if kind == "window":
        ring = 128 * rng.randint(8, 64)
        return {"kind": kind, "fmt": fmt, "layers": layers, "tokens": _log(rng, ring, 131072), "ntok": rng.randint(1, 4), "ring": ring,
                "window": rng.randint(ring // 4, ring - 8)}
    if kind == "sessions":
        shortest = _log(rng, 500, 4096)
        return {"kind": kind, "fmt": "f16", "layers": rng.randint(1, 4), "sessions": _log(rng, 2, 32), "shortest": shortest,
                "longest": _log(rng, shortest + 1000, 131072), "ntok": rng.randint(1, 4)}
    if kind == "prefill":
        if fmt == "f32":
            return {"kind": kind, "fmt": fmt, "layers": layers, "prefix": _log(rng, 16, 8192), "ntok": _log(rng, 5, 512), "q": "f32"}
        return {"kind": kind, "fmt": fmt, "layers": layers, "prefix": _log(rng, 16, 32768), "ntok": _log(rng, 5, 2048),
                "q": rng.choice(["f16", "f32"])}
    return {"kind": kind, "fmt": "f16", "layers": layers, "prefix": _log(rng, 500, 32768), "ntok": _log(rng, 8, 512), "q": rng.choice(["f16", "f32"])}


@functools.lru_cache(maxsize=None)
def _context(stream):
    """A host program has one context for all its caches."""
    return kv.KvContext(torch.cuda.current_device(), torch.cuda.current_stream())


def _room(n):
    return max(kv.CTX_MIN, (n + 1023) // 1024 * 1024)


def _lengths(case):
    """The sessions' lengths: evenly spread over the range, so that a pass's bytes are a property of the case."""
    n, lo, hi = case["sessions"], case["shortest"], case["longest"]
    return [lo + (hi - lo) * i // max(1, n - 1) + (i * 37) % 61 for i in range(n)]


class _State:
    pass


def _cache(s, case, g, tokens, room, ring=0):
    """A cache whose first `tokens` rows (all rows of a ring) are N(0,1)."""
    cache = kv.KvCache(s.ctx, kv.KvFormat.F16 if case["fmt"] == "f16" else kv.KvFormat.F32, case["layers"], _room(room), ring=ring)
    for l in range(case["layers"]):
        for t in cache.buffer_tensors(l):
            t[:ring or tokens].normal_(generator=g)
    cache.set_len(tokens)
    return cache


class _Rows:
    """Device memory of a cache as torch takes it over; a tensor made of it keeps the cache alive."""

    def __init__(self, cache, ptr, first, last):
        elem = cache.fmt.elem_bytes
        self.cache = cache
        self.__cuda_array_interface__ = {"shape": (last - first, kv.HKV, kv.D), "typestr": "<f%d" % elem, "version": 3, "strides": None,
                                         "data": (ptr + first * kv.ROW * elem, False)}


def _written(cache, layers, lo, hi):
    """The K and V rows [lo, hi) that a pass writes, layer by layer, where they lie in the cache."""
    rows = (lo % cache.ring, (hi - 1) % cache.ring + 1) if cache.ring else (lo, hi)
    if rows[0] >= rows[1]:  # the rows go over the ring's end
        rows = (0, cache.ring)
    return [torch.as_tensor(_Rows(cache, ptr, *rows), device="cuda") for l in range(layers) for ptr in cache.buffers(l)]


def prepare(case, seed):
    kind, L, n = case["kind"], case["layers"], case["ntok"]
    s = _State()
    s.case, s.kind = case, kind
    s.ctx = _context(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    if kind == "sessions":
        s.lens = _lengths(case)
        s.caches = [_cache(s, case, g, p, p + n) for p in s.lens]
        ns = len(s.lens)
        s.q = normal(L, ns, n, kv.HQ, kv.D)
        s.k, s.v = normal(ns, L, n, kv.HKV, kv.D), normal(ns, L, n, kv.HKV, kv.D)
        s.tabs = [torch.from_numpy(kv.rope_table(p, n)).cuda() for p in s.lens]
        s.out = torch.empty_like(s.q)
        s.parts = [[(c, p, l, q, o) for c, p, q, o in zip(s.caches, s.lens, s.q[l], s.out[l])] for l in range(L)]
        s.k, s.v = list(s.k), list(s.v)
        s.ctx.sync()
        return s

    s.pos = case["prefix"] if kind in ("prefill", "turn") else case["tokens"]
    s.cache = _cache(s, case, g, s.pos, s.pos + n, case.get("ring", 0))
    s.tab = torch.from_numpy(kv.rope_table(s.pos, n)).cuda()
    if kind == "step":
        s.qf, s.kb, s.vb = normal(L, n, kv.HQ, 2 * kv.D), normal(L, n, kv.HKV, kv.D), normal(L, n, kv.ROW)
        s.q_norm, s.k_norm = 1.0 + 0.1 * normal(L, kv.D), 1.0 + 0.1 * normal(L, kv.D)
        s.out = torch.empty(L, n, kv.HQ, kv.D, device="cuda", dtype=torch.float16)
    else:
        s.q = normal(L, n, kv.HQ, kv.D)
        if case.get("q") == "f16":
            s.q = s.q.half()
        s.k, s.v = normal(L, n, kv.HKV, kv.D), normal(L, n, kv.HKV, kv.D)
        s.out = torch.empty(L, n, kv.HQ, kv.D, device="cuda")
    if kind == "window":
        s.sinks = 2.0 * normal(L, kv.HQ)
    if kind == "turn":
        s.root = s.cache.read_root(s.pos)
        s.back = torch.empty((s.pos + n) * ROW_ELEMS * 2 * L, dtype=torch.uint8, pin_memory=True)
    s.rows = _written(s.cache, L, s.pos, s.pos + n)
    # each layer's tensors, as the layers around the attention hand them over
    s.parts = list(zip(s.qf, s.kb, s.vb, s.q_norm, s.k_norm, s.out) if kind == "step" else zip(s.q, s.out))
    if kind == "window":
        s.parts = list(zip(s.k, s.v, s.sinks, s.q, s.out))
    s.ctx.sync()
    return s


def run(s):
    if s.kind == "sessions":
        for cache, pos, k, v, tab in zip(s.caches, s.lens, s.k, s.v, s.tabs):
            cache.truncate(pos)  # the drafts that the step before had refused
            cache.append_layers(pos, k, v, tab)
        for parts in s.parts:
            s.ctx.attn_verify_batch([(cache, l, 0, pos, q, out) for cache, pos, l, q, out in parts])
        return [s.out]
    c, pos = s.cache, s.pos
    if s.kind == "verify":
        c.truncate(pos)
        c.append_layers(pos, s.k, s.v, s.tab)
        for l, (q, out) in enumerate(s.parts):
            c.attn_verify(l, 0, pos, q, out)
    elif s.kind == "step":
        c.truncate(pos)
        for l, (qf, kb, vb, q_norm, k_norm, out16) in enumerate(s.parts):
            c.attn_step(l, 0, pos, qf, kb, vb, q_norm, k_norm, s.tab, None, out16)
    elif s.kind == "window":
        c.truncate(pos)
        for l, (k, v, sinks, q, out) in enumerate(s.parts):
            c.append(l, pos, k, v, s.tab)
            c.attn_verify_window(l, s.case["window"], sinks, pos, q, out)
    elif s.kind == "prefill":
        c.truncate(pos)
        c.append_layers(pos, s.k, s.v, s.tab)
        for l, (q, out) in enumerate(s.parts):
            c.attn_prefill(l, 0, pos, q, out)
    else:
        c.truncate(0)
        c.write_root(s.root)
        c.append_layers(pos, s.k, s.v, s.tab)
        for l, (q, out) in enumerate(s.parts):
            c.attn_prefill(l, 0, pos, q, out)
        root = c.read_root(pos + s.case["ntok"], payload=s.back)
        return [s.out, root.payload]
    return [s.out] + s.rows


def work(case):
    """Bytes of the K and V rows, the queries, the new rows and the outputs, each once; the attention's multiplications and
    additions. A stored turn's bytes cross the host link twice as well."""
    L, n, kind = case["layers"], case["ntok"], case["kind"]
    elem = 2 if case["fmt"] == "f16" else 4
    row = ROW_ELEMS * elem
    per_key = 4 * kv.HQ * kv.D  # operations of one query token on one key, all heads

    if kind == "sessions":
        keys = [p + n for p in _lengths(case)]
        small = len(keys) * n * (2 * kv.HQ * kv.D * 4 + ROW_ELEMS * 4 + row)
        return {"bytes": L * (sum(keys) * row + small), "flops": L * n * per_key * sum(keys)}
    q_elem = 2 if case.get("q") == "f16" else 4
    pos = case["prefix"] if kind in ("prefill", "turn") else case["tokens"]
    keys = case["window"] + n - 1 if kind == "window" else pos + n
    seen = min(pos + n, keys)
    small = n * (kv.HQ * kv.D * (q_elem + 4) + ROW_ELEMS * 4 + row)
    if kind == "step":  # query and gate as f32, output as f16
        small = n * (kv.HQ * kv.D * (8 + 2) + ROW_ELEMS * 4 + row)
    flops = per_key * sum((case["window"] if kind == "window" else pos + t + 1) for t in range(n))
    total = seen * row + small
    if kind == "turn":
        total += pos * row + (pos + n) * row
    return {"bytes": L * total, "flops": L * flops}


def tolerance(case):
    """About four times what one layer's outputs show against the same attention in 64 bits: on the f16 cache, where queries and
    weights are rounded to f16, 2.2e-4 to 3.5e-4 (2-norm) and up to 1.7e-3 (largest difference); on the f32 cache 1.1e-6 and up to
    1.3e-5."""
    if case["fmt"] == "f32":
        return {"rel": 5e-6, "max": 6e-5}
    return {"rel": 1.4e-3, "max": 7e-3}
