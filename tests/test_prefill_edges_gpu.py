"""The tensor-core prefill at the edges of its KV tiles (64 tokens) and query tiles (128 rows), where the items of a short call
have one tile, an odd or an even number of them, or a half of the block without any."""
import math

import numpy as np
import pytest
import torch

import oracle
from tinycoder_inference_b200 import ops
from tests.util import assert_close, dev, host

pytestmark = pytest.mark.gpu


def _check(S, pos, nH, nKV, hd):
    r = np.random.default_rng(S + pos + hd)
    q, k, v = (r.standard_normal((n, h, hd), dtype=np.float32) for n, h in ((S, nH), (pos + S, nKV), (pos + S, nKV)))
    out = torch.full((S + 1, nH, hd), float("nan"), device="cuda")
    n = ops.prefill_f16_scratch_bytes(S, nH, nKV, hd, cachePos=pos)
    scratch = torch.empty(n + 1024, dtype=torch.uint8, device="cuda")
    off = (-scratch.data_ptr()) % 1024
    ops.prefill_f16(dev(q), dev(k), dev(v), out[:S], scratch[off:off + n], S, nH, nKV, hd, cachePos=pos)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    q, k, v = (x.astype(np.float16) for x in (q, k, v))
    want = oracle.attention_f64(q.astype(np.float32), k, v, None, None, S, nH, nKV, hd, pos, 1.0 / math.sqrt(hd))
    # probabilities are rounded to fp16 (2^-11 each, both in the sums): 2^-10 of the largest |v| of N(0, 1) rows (4.5)
    assert_close(host(out[:S]), want, rtol=0.0, atol=4.5e-3, what=f"{S} rows behind {pos}")
    assert torch.isnan(out[S]).all()


def _check_norm(S, pos, nH, nKV, hd, peak=None):
    """Against the distance that the fp16 probabilities explain: each is off by at most 2^-11 of itself, 2^-11 / sqrt(3) on
    average and independently of the others, and so is then the output of a row and head -- 2.8e-4 of its norm where the
    values are N(0, 1).  Four times that.  A weight of a block's results that is off by more than a few thousandths shows."""
    r = np.random.default_rng(7 * S + pos + hd)
    q, k, v = (r.standard_normal((n, h, hd), dtype=np.float32) for n, h in ((S, nH), (pos + S, nKV), (pos + S, nKV)))
    if peak is not None:    # a share of q that all rows have in common, and keys that lie along it
        log2, rows = peak
        u = np.where(r.random(hd) < 0.5, -1.0, 1.0).astype(np.float32)
        q += 0.5 * u
        k[rows] += np.float32(log2 * math.log(2.0) / math.sqrt(hd) / 0.5) * u
    q, k, v = (x.astype(np.float16) for x in (q, k, v))
    out = torch.full((S, nH, hd), float("nan"), device="cuda")
    n = ops.prefill_f16_scratch_bytes(S, nH, nKV, hd, cachePos=pos)
    scratch = torch.empty(n + 1024, dtype=torch.uint8, device="cuda")
    off = (-scratch.data_ptr()) % 1024
    ops.prefill_f16(*(dev(x.astype(np.float32)) for x in (q, k, v)), out, scratch[off:off + n], S, nH, nKV, hd, cachePos=pos)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    want = oracle.attention_f64(q.astype(np.float32), k, v, None, None, S, nH, nKV, hd, pos, 1.0 / math.sqrt(hd)).astype(np.float64)
    err = np.linalg.norm(host(out) - want, axis=2) / np.linalg.norm(want, axis=2)
    assert err.max() < 4 * 2.0 ** -11 / math.sqrt(3.0), (err.max(), np.unravel_index(err.argmax(), err.shape))


@pytest.mark.parametrize("S,pos", [(1, 0), (63, 0), (64, 0), (65, 0), (2, 127), (128, 64), (129, 63), (257, 190)])
@pytest.mark.parametrize("nH,nKV,hd", [(7, 1, 64), (6, 2, 128), (4, 2, 256)])
def test_tile_edges(S, pos, nH, nKV, hd):
    _check(S, pos, nH, nKV, hd)


# few items: clusters of 8, 4 and 2 blocks share an item's KV tiles; ragged rows, KV tiles that do not divide evenly, rows
# whose blocks have no tile at all (no prefix, long calls) or only tiles behind their diagonal
@pytest.mark.parametrize("S,pos,nH,nKV,hd", [(1, 3000, 14, 2, 64), (100, 1500, 8, 4, 64), (385, 1900, 8, 4, 64), (512, 1600, 14, 2, 64),
                                             (77, 1217, 12, 2, 128), (1100, 0, 3, 1, 128), (512, 777, 8, 2, 128),
                                             (130, 2500, 28, 4, 128), (77, 1500, 2, 1, 256), (1000, 0, 4, 2, 256),
                                             (300, 601, 16, 2, 256)])
def test_items_shared_by_a_cluster(S, pos, nH, nKV, hd):
    _check(S, pos, nH, nKV, hd)
    _check_norm(S, pos, nH, nKV, hd)


# A few keys in one KV tile outweigh all others, by 2^30 or so far that what the other tiles add vanishes: the maxima of the
# blocks (and of the even and odd tiles of a block) that share an item are then far apart.  Tile 0 is the first block's, tile 7 the
# last one's whether 2, 4 or 8 blocks share the tiles.
@pytest.mark.parametrize("tile", [0, 7])
@pytest.mark.parametrize("log2", [30, 150])
@pytest.mark.parametrize("S,pos,nH,nKV,hd", [(16, 3000, 14, 2, 64), (77, 1217, 12, 2, 128), (130, 2500, 28, 4, 128), (300, 601, 16, 2, 256),
                                             (1000, 0, 4, 2, 256)])
def test_items_shared_by_a_cluster_with_keys_that_dominate(S, pos, nH, nKV, hd, log2, tile):
    _check_norm(S, pos, nH, nKV, hd, (log2, [64 * tile + i for i in (3, 17, 60)]))


# The launch in front of the attention: q and K / V in blocks of their own (up to two of each per SM, and no more for the
# rows that the store already has than for q) or one after the other in every block; the sizes lie on both sides of each of the two lines on 148 SMs.
@pytest.mark.parametrize("mode,nH,nKV,hd,before,rows", [("f32", 28, 4, 128, 0, 169), ("f32", 28, 4, 128, 0, 170), ("f32+i8", 28, 4, 128, 0, 169),
                                                        ("i8", 28, 4, 128, 3, 170), ("f32", 8, 2, 128, 200, 100), ("i8", 8, 2, 128, 204, 100),
                                                        ("f16", 14, 2, 64, 5, 676), ("f16", 14, 2, 64, 0, 679), ("f32", 4, 4, 256, 76, 75),
                                                        ("f32", 4, 4, 256, 80, 75)])
def test_prompt_rows_in_either_kind_of_launch(mode, nH, nKV, hd, before, rows):
    n, inv = before + rows, 1.0 / math.sqrt(hd)
    r = np.random.default_rng(n + hd)
    q, k, v = (r.standard_normal((n, h, hd), dtype=np.float32) for h in (nH, nKV, nKV))
    rope = oracle.rope_tables(n, hd, 1e6) if mode in ("f32", "f16") else None
    s = ops.KvSession(nH, nKV, hd, n, 1, mode=mode, rope=None if rope is None else tuple(dev(t) for t in rope), prefill_scratch_rows=n)
    for a, b in ((0, before), (before, n)):
        if a == b:
            continue
        dq, out = dev(q[a:b]), torch.full((b - a, nH, hd), float("nan"), device="cuda")
        s.attend(0, dq, dev(k[a:b]), dev(v[a:b]), out, a)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    K, V, q = np.zeros_like(k), np.zeros_like(v), q[before:]
    if rope is not None:
        q = oracle.rope_q(q, *rope, rows, nH, hd, before)
        oracle.kv_append(k, v, K, V, n, nKV, hd, 0, ropePos=0, cosT=rope[0], sinT=rope[1])
    else:
        K, V = k, v
    assert np.array_equal(host(dq), q)
    if mode != "i8":
        dt = np.float16 if mode == "f16" else np.float32
        assert np.array_equal(host(s.kvK[0]), K.astype(dt)) and np.array_equal(host(s.kvV[0]), V.astype(dt))
    if "i8" in mode:
        quant = oracle.quant_kv8(K, V, nKV, hd)
        for have, want in zip((s.k8, s.v8, s.ks, s.vs), quant):
            assert np.array_equal(host(have[0, :n]), want)
    if mode == "i8":    # the rows as the store holds them
        K, V = (x8.astype(np.float32) * sc[:, :, None] for x8, sc in ((quant[0], quant[2]), (quant[1], quant[3])))
    q, K, V = (x.astype(np.float16) for x in (q, K, V))
    want = oracle.attention_f64(q.astype(np.float32), K, V, None, None, rows, nH, nKV, hd, before, inv)
    assert_close(host(out), want, rtol=0.0, atol=4.5e-3, what=f"{rows} rows behind {before}")
