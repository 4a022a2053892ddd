"""The launches that take a token's new row along, at the sizes where their splits change: tile and stream edges, one and
several clusters, blocks without rows, more than eight q heads per kv head."""
import math

import numpy as np
import pytest
import torch

import oracle
from tinycoder_inference_b200 import ops
from tests.util import assert_close, dev, host

pytestmark = pytest.mark.gpu


def _rows(seed, nH, nKV, hd, n):
    r = np.random.default_rng(seed)
    return (r.standard_normal((1, nH, hd), dtype=np.float32), r.standard_normal((n, nKV, hd), dtype=np.float32),
            r.standard_normal((n, nKV, hd), dtype=np.float32))


def _int8_session(nH, nKV, hd, ctx, window, seed):
    """A session on the int8 store whose rows [0, ctx) are written; the token's q / k / v; everything quantised."""
    q, k, v = _rows(seed, nH, nKV, hd, ctx + 1)
    s = ops.KvSession(nH, nKV, hd, window, 1, mode="i8")
    if ctx:
        ops.kv_quantize_i8(dev(k[:ctx]), dev(v[:ctx]), s.k8[0], s.v8[0], s.ks[0], s.vs[0], ctx, nKV, hd)
    return s, q, k, v, oracle.quant_kv8(k, v, nKV, hd)


# tiles of 32 tokens (head_dim 128) / 16 (head_dim 256), eight streams, sixteen tiles of a stream in flight
@pytest.mark.parametrize("nH,nKV,hd,ctx", [(28, 4, 128, 0), (28, 4, 128, 31), (28, 4, 128, 32), (8, 2, 128, 255),
                                           (12, 2, 128, 256), (28, 4, 128, 2047), (28, 4, 128, 4096), (9, 1, 128, 4129),
                                           (28, 4, 128, 9000), (16, 2, 256, 0), (16, 2, 256, 15), (16, 4, 256, 128),
                                           (8, 4, 256, 2049), (20, 2, 256, 4500),
                                           (72, 1, 128, 300)])
def test_captured_step_on_the_int8_store(nH, nKV, hd, ctx):
    """The device-position step stores the row itself and keeps the causal kernel's accumulation order."""
    s, q, k, v, quant = _int8_session(nH, nKV, hd, ctx, ctx + 300, seed=ctx + hd + nH)
    out = torch.full((1, nH, hd), float("nan"), device="cuda")
    pos = torch.tensor([ctx], dtype=torch.int32, device="cuda")
    s.attend(0, dev(q), dev(k[ctx:]), dev(v[ctx:]), out, ctx, dev_pos=pos, graph_capture=True)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    for have, want in zip((s.k8, s.v8, s.ks, s.vs), quant):
        assert np.array_equal(host(have[0, :ctx + 1]), want)
    causal = torch.full((1, nH, hd), float("nan"), device="cuda")
    ops.prefill_i8(dev(q), s.k8[0], s.v8[0], s.ks[0], s.vs[0], causal, 1, nH, nKV, hd, ctx)
    # the same products in the same order: what is left is the order of the last eight additions (2^-24 each)
    assert_close(host(out), host(causal), rtol=1e-6, atol=1e-6, what="captured step against the causal kernel")
    want = oracle.attention_i8(q, *quant, 1, nH, nKV, hd, ctx, 1.0 / math.sqrt(hd))
    assert_close(host(out), want, what="captured step against the oracle")


# head_dim 128: 128-token tiles, clusters of 2 .. 16 blocks, then blocks and a merge; head_dim 256: chunks and a merge
@pytest.mark.parametrize("mode", ["i8", "f32+i8"])
@pytest.mark.parametrize("nH,nKV,hd,ctx", [(28, 4, 128, 127), (28, 4, 128, 128), (28, 4, 128, 1151), (40, 8, 128, 2048),
                                           (9, 1, 128, 1500), (28, 4, 128, 9500), (16, 2, 256, 64), (16, 2, 256, 1100),
                                           (20, 2, 256, 3000)])
def test_eager_step_on_an_int8_pool(mode, nH, nKV, hd, ctx):
    q, k, v = _rows(ctx + nH, nH, nKV, hd, ctx + 1)
    s = ops.KvSession(nH, nKV, hd, ctx + 40, 2, mode=mode)
    if mode == "i8":
        ops.kv_quantize_i8(dev(k[:ctx]), dev(v[:ctx]), s.k8[1], s.v8[1], s.ks[1], s.vs[1], ctx, nKV, hd)
    else:
        ops.kv_append(dev(k[:ctx]), dev(v[:ctx]), s.kvK[1], s.kvV[1], ctx, nKV, hd, 0)
    out = torch.full((1, nH, hd), float("nan"), device="cuda")
    s.attend(1, dev(q), dev(k[ctx:]), dev(v[ctx:]), out, ctx)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    quant = oracle.quant_kv8(k, v, nKV, hd)
    for have, want in zip((s.k8, s.v8, s.ks, s.vs), quant):
        assert np.array_equal(host(have[1, :ctx + 1]), want)
    if mode != "i8":
        assert np.array_equal(host(s.kvK[1, :ctx + 1]), k) and np.array_equal(host(s.kvV[1, :ctx + 1]), v)
    want = oracle.attention_i8(q, *quant, 1, nH, nKV, hd, ctx, 1.0 / math.sqrt(hd))
    assert_close(host(out), want, what=f"{mode} eager step")


# 16-token tiles; one block, one cluster, blocks and a merge; host and device position
@pytest.mark.parametrize("dev_pos", [False, True])
@pytest.mark.parametrize("mode,nH,nKV,hd,ctx", [("f32", 14, 2, 64, 0), ("f32", 14, 2, 64, 15), ("f32", 14, 2, 64, 2047),
                                                ("f32", 9, 1, 128, 640), ("f32", 28, 4, 128, 5000), ("f16", 14, 2, 64, 16),
                                                ("f16", 28, 4, 128, 129), ("f16", 28, 4, 128, 2500), ("f16", 40, 2, 128, 9001),
                                                ("f16", 14, 2, 64, 20000),
                                                # (head_dim 256: a rotation partner in the lane's other float4, six warps for
                                                # eight columns; groups of 3, 8 and 20; one tile, a cluster, a merge)
                                                ("f32", 3, 1, 256, 0), ("f32", 16, 2, 256, 0), ("f32", 6, 2, 256, 700),
                                                ("f32", 20, 1, 256, 333), ("f32", 16, 2, 256, 15000), ("f32", 20, 1, 256, 9000)])
def test_rotating_step_on_an_f32_or_fp16_store(mode, nH, nKV, hd, ctx, dev_pos):
    q, k, v = _rows(ctx + hd, nH, nKV, hd, ctx + 1)
    cos, sin = oracle.rope_tables(ctx + 1, hd, 1e6)
    s = ops.KvSession(nH, nKV, hd, ctx + 1, 1, mode=mode, rope=(dev(cos), dev(sin)))
    dt = np.float16 if mode == "f16" else np.float32
    if ctx:
        s.kvK[0, :ctx].copy_(dev(k[:ctx].astype(dt)))
        s.kvV[0, :ctx].copy_(dev(v[:ctx].astype(dt)))
    out, dq = torch.full((1, nH, hd), float("nan"), device="cuda"), dev(q)
    pos = torch.tensor([ctx], dtype=torch.int32, device="cuda") if dev_pos else None
    s.attend(0, dq, dev(k[ctx:]), dev(v[ctx:]), out, ctx, dev_pos=pos, graph_capture=dev_pos)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    qr = oracle.rope_q(q, cos, sin, 1, nH, hd, ctx)
    kk, vv = np.zeros((ctx + 1, nKV, hd), np.float32), np.zeros((ctx + 1, nKV, hd), np.float32)
    oracle.kv_append(k[ctx:], v[ctx:], kk, vv, 1, nKV, hd, ctx, ropePos=ctx, cosT=cos, sinT=sin)
    kk[:ctx], vv[:ctx] = k[:ctx], v[:ctx]
    kk, vv = kk.astype(dt), vv.astype(dt)
    assert np.array_equal(host(dq), qr)
    assert np.array_equal(host(s.kvK[0]), kk) and np.array_equal(host(s.kvV[0]), vv)
    assert_close(host(out), oracle.attention_kv(qr, kk, vv, 1, nH, nKV, hd, ctx, 1.0 / math.sqrt(hd)), what=f"{mode} step")


# (window 40000: several blocks per kv head and a merge, which rotates q by the position as well)
@pytest.mark.parametrize("mode,nH,nKV,hd,window", [("i8", 28, 4, 128, 64), ("i8", 16, 2, 256, 64), ("f32", 14, 2, 64, 64),
                                                   ("f16", 28, 4, 128, 64), ("f16", 28, 4, 128, 40000)])
@pytest.mark.parametrize("at", [0xffffffff, 0x80000000, 50000])
def test_a_device_position_outside_the_store_writes_no_row(mode, nH, nKV, hd, window, at):
    """(0xffffffff: position + 1 wraps to a length of 0)"""
    q, k, v = _rows(hd, nH, nKV, hd, 1)
    rope = tuple(dev(t) for t in oracle.rope_tables(window, hd, 1e6)) if mode[0] == "f" else None
    s = ops.KvSession(nH, nKV, hd, window, 2, mode=mode, rope=rope)
    stores = [t for t in (getattr(s, n, None) for n in ("kvK", "kvV", "k8", "v8", "ks", "vs")) if t is not None]
    before = [t.clone() for t in stores]
    pos = torch.from_numpy(np.array([at], np.uint32).view(np.int32)).cuda()
    s.attend(1, dev(q), dev(k), dev(v), torch.zeros((1, nH, hd), device="cuda"), 3, dev_pos=pos, graph_capture=True)
    torch.cuda.synchronize()
    assert ops.device_status(raise_on_flags=False) == 32
    for have, want in zip(stores, before):
        assert torch.equal(torch.nan_to_num(have.float()), torch.nan_to_num(want.float()))


@pytest.mark.parametrize("nH,nKV,hd,ctx,growth", [(28, 4, 128, 300, 0.0), (28, 4, 128, 4600, 6.0), (14, 2, 128, 4100, 0.4), (16, 2, 256, 2700, 6.0),
                                                  (8, 4, 256, 1500, 0.4)])
def test_captured_int8_step_accumulates_like_causal_rows(nH, nKV, hd, ctx, growth):
    """The launch a captured step replays keeps the causal kernel's roundings over several rounds of tiles, where no tile moves a
    head's reference point or the bound of the V scales, where all of them do, and where some do: scores and V rows that grow with the
    position, by `growth` powers of two in 16 rows."""
    g = torch.Generator(device="cuda").manual_seed(ctx)
    s = ops.KvSession(nH, nKV, hd, ctx + 100, 1, mode="i8")
    q = torch.randn((1, nH, hd), device="cuda", generator=g)
    k, v = (torch.randn((ctx, nKV, hd), device="cuda", generator=g) for _ in range(2))
    at = torch.arange(ctx, device="cuda", dtype=torch.float32)[:, None, None] / 16.0 * growth
    mean = q.view(nKV, nH // nKV, hd).mean(1)
    k += at * math.log(2.0) * math.sqrt(hd) * mean / (mean * mean).sum(1, keepdim=True)
    v *= torch.exp2(torch.clamp(at / 6.0, max=40.0))
    ops.kv_quantize_i8(k[:-1].contiguous(), v[:-1].contiguous(), s.k8[0], s.v8[0], s.ks[0], s.vs[0], ctx - 1, nKV, hd)
    out, want = torch.empty_like(q), torch.empty_like(q)
    s.attend(0, q, k[-1:].contiguous(), v[-1:].contiguous(), out, ctx - 1, dev_pos=torch.tensor([ctx - 1], dtype=torch.int32, device="cuda"))
    ops.prefill_i8(q, s.k8[0], s.v8[0], s.ks[0], s.vs[0], want, 1, nH, nKV, hd, ctx - 1)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    # the eight streams' results are put together in another order: a handful of f32 roundings
    assert float((out - want).norm() / want.norm()) < 1e-6
