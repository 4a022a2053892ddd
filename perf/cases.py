"""The work this library is timed on: the attention block as a program drives it, over the
range of shapes, stores and options it is built for.

Four paths, all through `tinycoder_inference_b200.ops`:

  decode    one new token through `layers` KV slots of a `KvSession` (eager calls, position on
            the host): store the token's K/V row, attend over everything before it
  replay    the same step with the position on the device, captured once in a CUDA graph -- the
            handle a serving program keeps -- and replayed
  prompt    a fresh prompt: `KvSession.clear`, then the prompt in calls of at most `chunk` rows
            through every slot (`scratch` says whether the session has room for the fp16 twins;
            without it the exact f32 causal kernels run)
  batch     one decode step of `batch` sequences that share an int8 pool per layer
            (`ops.decode_i8_batch`), the new tokens' rows handed in; `ragged` lengths live on the
            device

and three kinds of model in front of them:

  dense     rotation tables in the session: K (and q, in place) are rotated by the store
  plain     rows arrive rotated (the int8 and mirrored stores take them like that)
  gated     Q/K RMSNorm + partial rotation in front, sigmoid gate behind (head_dim 256 models)
"""
from __future__ import annotations

import math
import random

import torch

from tinycoder_inference_b200 import ops

# (q heads, kv heads) per head_dim: the shapes of the benchmark, the planner's models and the tests
SHAPES = {64: [(14, 2), (8, 4)], 128: [(28, 4), (12, 2), (40, 8), (8, 2)], 256: [(16, 2), (16, 4), (8, 4)]}
ROPE_THETA = 1e6
GATED_DIMS, GATED_THETA = 64, 1e7     # rotated dims and base of the gated models
# no drawn case is larger than the largest listed ones
MAX_BYTES, MAX_FLOPS, MAX_EXACT_FLOPS = 1.2e9, 3.0e11, 2.0e10


def _case(name, path, model, store, heads, kv_heads, head_dim, ctx, rows=1, layers=1, **more):
    c = {"name": name, "path": path, "model": model, "store": store, "q_heads": heads, "kv_heads": kv_heads,
         "head_dim": head_dim, "ctx": ctx, "rows": rows, "layers": layers}
    c.update(more)
    return c


def listed():
    return [
        # one attention layer of a small dense model at a 2048-row context: the smallest call, a
        # completion model in an editor; latency and launches are all there is
        _case("decode_f32_small", "decode", "dense", "f32", 14, 2, 64, ctx=2047),
        # a token of a dense model on the fp16 cache, a chat some thousand tokens in
        _case("decode_f16", "decode", "dense", "f16", 28, 4, 128, ctx=8191, layers=4),
        # f32 store with the int8 decode mirror (the planner's first choice), an odd position
        _case("decode_mirror", "decode", "plain", "f32+i8", 28, 4, 128, ctx=4098, layers=8),
        # a gated model with int8 as its store and a long context: norm + rotation, attention, gate
        _case("decode_gated_i8", "decode", "gated", "i8", 16, 2, 256, ctx=16383, layers=8),
        # the engine's captured decode step on the int8 store: position on the device, replayed
        _case("replay_i8", "replay", "plain", "i8", 28, 4, 128, ctx=5000, layers=8, window=8192),
        # one long session of a 7B-shaped model, all its layers, new rows quantised by the launch
        _case("batch1_long", "batch", "plain", "i8", 28, 4, 128, ctx=32767, layers=28, batch=1, ragged=False),
        # eight sessions in step (batched serving)
        _case("batch8", "batch", "plain", "i8", 28, 4, 128, ctx=8191, layers=8, batch=8, ragged=False),
        # a serving mix: 64 sessions with lengths anywhere in [512, 32768]
        _case("batch64_ragged", "batch", "plain", "i8", 28, 4, 128, ctx=32767, layers=1, batch=64, ragged=True),
        # a whole prompt in one call, f32 store + int8 mirror, on the tensor cores
        _case("prompt_4096", "prompt", "plain", "f32+i8", 28, 4, 128, ctx=0, rows=4096, layers=2, chunk=4096,
              scratch=True),
        # a prompt fed in the engine's 512-row calls, int8 store, a ragged last call
        _case("prompt_chunked", "prompt", "plain", "i8", 28, 4, 128, ctx=0, rows=1900, layers=2, chunk=512,
              scratch=True),
        # a short instruction to a gated model on its f32 store
        _case("prompt_gated", "prompt", "gated", "f32", 16, 2, 256, ctx=0, rows=333, layers=4, chunk=512, scratch=True),
        # a session without scratch for the twins: exact f32 causal attention
        _case("prompt_exact", "prompt", "dense", "f32", 14, 2, 64, ctx=0, rows=512, layers=2, chunk=512, scratch=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    while True:
        path = rng.choice(["decode", "decode", "decode", "replay", "batch", "batch", "prompt", "prompt", "prompt"])
        layers = rng.choice([1, 2, 4, 8])
        if path == "batch":
            model, store, hd = "plain", "i8", 128
        else:
            model, store, hd = rng.choice([("dense", "f32", 64), ("dense", "f32", 128), ("dense", "f16", 64),
                                           ("dense", "f16", 128), ("plain", "f32+i8", 128), ("plain", "i8", 128),
                                           ("gated", "f32", 256), ("gated", "f32+i8", 256), ("gated", "i8", 256)])
        heads, kv = rng.choice(SHAPES[hd])
        c = {"path": path, "model": model, "store": store, "q_heads": heads, "kv_heads": kv, "head_dim": hd,
             "layers": layers}
        if path in ("decode", "replay"):
            c.update(ctx=_log(rng, 16, 65536 if path == "decode" else 16384), rows=1)
            if path == "replay":
                c["window"] = -(-(c["ctx"] + 1) * rng.choice([1, 2]) // 1024) * 1024
        elif path == "batch":
            c.update(ctx=_log(rng, 64, 131072), rows=1, batch=_log(rng, 1, 64))
            c["ragged"] = c["batch"] > 1 and rng.random() < 0.5
        else:
            c.update(ctx=0, rows=_log(rng, 8, 4096), chunk=rng.choice([512, 512, 4096]), scratch=rng.random() < 0.7)
        w = work(c)
        small = c.get("scratch", True) or w["flops"] <= MAX_EXACT_FLOPS
        if w["bytes"] <= MAX_BYTES and w["flops"] <= MAX_FLOPS and small:
            return c


# ---- what a program holds before the call ----------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _tables(rows, hd, gated):
    t = ops.mrope_tables(rows, GATED_DIMS, GATED_THETA) if gated else ops.rope_tables(rows, hd, ROPE_THETA)
    return tuple(torch.from_numpy(x).cuda() for x in t)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _quantise_random(g, k8, v8, ks, vs, rows, kv, hd):
    """Fills pool rows [0, rows) the way a prompt does: N(0, 1) rows through the quantiser."""
    step = 1 << 17
    for a in range(0, rows, step):
        n = min(step, rows - a)
        ops.kv_quantize_i8(_randn(g, n, kv, hd), _randn(g, n, kv, hd), k8, v8, ks, vs, n, kv, hd, dst_base=a)


def _prepare_session(case, g):
    heads, kv, hd = case["q_heads"], case["kv_heads"], case["head_dim"]
    layers, rows, ctx = case["layers"], case["rows"], case["ctx"]
    window = case.get("window") or -(-(ctx + rows) // 1024) * 1024
    gated = case["model"] == "gated"
    tables = None if case["model"] == "plain" else _tables(window, hd, gated)
    chunk = min(case.get("chunk", 1), rows)
    s = ops.KvSession(heads, kv, hd, window, layers, mode=case["store"],
                      rope=tables if case["model"] == "dense" else None,
                      prefill_scratch_rows=chunk if case.get("scratch") else 0)
    st = {"case": case, "s": s, "tables": tables}
    if ctx:
        if case["store"] == "i8":
            for l in range(layers):
                _quantise_random(g, s.k8[l], s.v8[l], s.ks[l], s.vs[l], ctx, kv, hd)
        else:
            s.kvK[:, :ctx].normal_(generator=g)
            s.kvV[:, :ctx].normal_(generator=g)
    st["k"], st["v"] = _randn(g, layers, rows, kv, hd), _randn(g, layers, rows, kv, hd)
    out = torch.zeros((layers, rows, heads, hd), device="cuda")
    if gated:
        st["qg"] = _randn(g, layers, rows, heads, 2 * hd)
        st["q"] = torch.zeros((layers, rows, heads, hd), device="cuda")
        st["wq"], st["wk"] = 1.0 + 0.1 * _randn(g, hd), 1.0 + 0.1 * _randn(g, hd)
    else:
        st["q"] = _randn(g, layers, rows, heads, hd)
    # what a call of the pass is handed, per piece of the prompt and per layer
    st["calls"] = []
    for a in range(0, rows, chunk):
        n = min(chunk, rows - a)
        st["calls"].append((n, [tuple(t[l, a:a + n] for t in (st["q"], st["k"], st["v"], out)) +
                                ((st["qg"][l, a:a + n],) if gated else ()) for l in range(layers)]))
    if ctx > 1 and case["path"] == "decode":
        # the token before this one has been decoded already (its row replaces the last filled one)
        for l in range(layers):
            one = [_randn(g, 1, h, hd) for h in (heads, kv, kv, heads)]
            s.attend(l, *one, ctx - 1)
    if ctx:
        s.commit(ctx)
    pools = [t for t in (getattr(s, n, None) for n in ("kvK", "kvV", "k8", "v8", "ks", "vs")) if t is not None]
    st["result"] = [out] + pools
    if case["model"] == "dense":
        st["result"].append(st["q"])
    if gated:
        st["result"].append(st["k"])
    if case["path"] == "replay":
        pos = torch.tensor([ctx], dtype=torch.int32, device="cuda")
        st["pos"] = pos
        # a graph is captured after one eager call; that call's effect on q and K is undone
        keep = [st["q"].clone(), st["k"].clone()]
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _layers(st, 1, st["calls"][0][1], ctx, pos, True)
        torch.cuda.current_stream().wait_stream(side)
        st["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(st["graph"]):
            _layers(st, 1, st["calls"][0][1], ctx, pos, True)
        st["q"].copy_(keep[0])
        st["k"].copy_(keep[1])
    return st


def _prepare_batch(case, g):
    heads, kv, hd = case["q_heads"], case["kv_heads"], case["head_dim"]
    layers, batch, ctx = case["layers"], case["batch"], case["ctx"]
    st = {"case": case}
    if case["ragged"]:
        # lengths spread evenly over [max / 64, max], in the seed's order; every sequence's rows are
        # contiguous in the pool
        lo, hi = max(1, (ctx + 1) // 64), ctx + 1
        u = (torch.arange(batch, device="cuda") + torch.rand(batch, generator=g, device="cuda")) / batch
        lens = (lo + (u * (hi + 1 - lo)).long().clamp_(max=hi - lo))[torch.randperm(batch, generator=g, device="cuda")]
        st["lens"] = lens.to(torch.int32)
        st["base"] = torch.cumsum(lens, 0) - lens
        total = int(lens.sum())
        rows = batch * lo + (batch + 1) * (hi + 1 - lo) // 2 + batch    # room for any draw of lengths
    else:
        st["lens"] = st["base"] = None
        total = rows = batch * (ctx + 1)
    st["k8"] = torch.zeros((layers, rows + 16, kv, hd), dtype=torch.int8, device="cuda")
    st["v8"] = torch.zeros_like(st["k8"])
    st["ks"] = torch.zeros((layers, rows + 16, kv), device="cuda")
    st["vs"] = torch.zeros_like(st["ks"])
    for l in range(layers):
        _quantise_random(g, st["k8"][l], st["v8"][l], st["ks"][l], st["vs"][l], total, kv, hd)
    _, slots = ops.split_geometry(ctx + 1, heads, hd)
    st["slots"] = slots if batch == 1 else min(slots, 64)
    st["ws"] = ops.workspace(batch, heads, hd, st["slots"])
    q = _randn(g, layers, batch, heads, hd)
    k, v = _randn(g, layers, batch, kv, hd), _randn(g, layers, batch, kv, hd)
    out = torch.zeros_like(q)
    st["layers"] = [dict(q=q[l], out=out[l], new=(k[l], v[l]), pool=tuple(st[n][l] for n in ("k8", "v8", "ks", "vs")),
                         after=(st["k8"][(l + 1) % layers], st["v8"][(l + 1) % layers])) for l in range(layers)]
    st["result"] = [out, st["k8"], st["v8"], st["ks"], st["vs"]]
    return st


def prepare(case, seed):
    g = _gen(seed)
    return _prepare_batch(case, g) if case["path"] == "batch" else _prepare_session(case, g)


# ---- one pass ------------------------------------------------------------------------------

def _layers(st, n, calls, pos, dev_pos=None, graph_capture=False):
    c, s = st["case"], st["s"]
    if c["model"] == "gated":
        heads, kv, hd = c["q_heads"], c["kv_heads"], c["head_dim"]
        cos, sin = st["tables"]
        for l, (q, k, v, out, qg) in enumerate(calls):
            ops.qk_norm_rope(qg, q, k, st["wq"], st["wk"], hd, GATED_DIMS, heads, kv, n, pos, cos, sin, dev_pos=dev_pos)
            s.attend(l, q, k, v, out, pos, dev_pos=dev_pos, graph_capture=graph_capture)
            ops.sigmoid_gate(out, qg, n, heads, hd)
    else:
        for l, (q, k, v, out) in enumerate(calls):
            s.attend(l, q, k, v, out, pos, dev_pos=dev_pos, graph_capture=graph_capture)


def run(st):
    c = st["case"]
    if c["path"] == "replay":
        st["graph"].replay()
    elif c["path"] == "decode":
        # (the position is not committed: every pass decodes the same token)
        _layers(st, 1, st["calls"][0][1], st["s"].begin(1))
    elif c["path"] == "prompt":
        s = st["s"]
        s.clear()
        for n, calls in st["calls"]:
            _layers(st, n, calls, s.begin(n))
            s.commit(n)
    else:
        uniform = not c["ragged"]
        for x in st["layers"]:
            k8, v8, ks, vs = x["pool"]
            ops.decode_i8_batch(x["q"], k8, v8, ks, vs, x["out"], st["ws"], st["lens"], c["batch"], c["q_heads"],
                                c["kv_heads"], c["head_dim"], c["ctx"] + 1, st["slots"],
                                rows_per_seq=c["ctx"] + 1 if uniform else 0, row_base=st["base"], pdl=True,
                                prefetch_rows=c["ctx"] if uniform else 0, next_kv=x["after"], append=x["new"])
    return st["result"]


# ---- what a pass cannot do without -----------------------------------------------------------

def _row_bytes(kind, hd):
    """K and V of one row and kv head."""
    return {"f32": 8 * hd, "f16": 4 * hd, "i8": 2 * (hd + 4)}[kind]


def work(case):
    heads, kv, hd, rows, layers = (case[k] for k in ("q_heads", "kv_heads", "head_dim", "rows", "layers"))
    batch = case.get("batch", 1)
    gated = case["model"] == "gated"
    # q (q and gate in the gated models), the output, the new K/V rows
    io = 4 * batch * rows * (heads * hd * (3 if gated else 2) + 2 * kv * hd)
    if case["path"] == "prompt":
        stores = {"f32": ["f32"], "f16": ["f16"], "i8": ["i8"], "f32+i8": ["f32", "i8"]}[case["store"]]
        kvb = rows * kv * sum(_row_bytes(s, hd) for s in stores)
        flops = 2 * hd * heads * rows * (rows + 1)
    else:
        n = case["ctx"] + 1
        total = batch * n
        if case.get("ragged"):
            total = batch * (max(1, n // 64) + n) // 2
        read = case["store"]
        if read == "f32+i8":
            read = "f32" if case["path"] == "replay" else "i8"
        kvb = total * kv * _row_bytes(read, hd)
        flops = 4 * hd * heads * total
    return {"bytes": float(layers * (io + kvb)), "flops": float(layers * flops)}


def tolerance(case):
    # f32 results.  The prompt on the tensor cores rounds q, K, V and the probabilities to fp16
    # (2^-11 each); everything else keeps at least 21 bits of every operand and sums in f32.
    if case["path"] == "prompt" and case["scratch"]:
        return {"rel": 2e-3, "max": 2e-2}
    return {"rel": 1e-5, "max": 1e-3}
