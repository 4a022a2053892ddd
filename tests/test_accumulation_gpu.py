"""How far the f32 / fp16 paths are from a 64-bit evaluation.  A tensor-core product drops the bits of its running sum that
do not fit (up to 2^-23 of it, always towards zero), so a path that adds thousands of tokens into one accumulator drifts;
the kernels add short chains of products in f32 instead.  The bounds: 2^-24 relative per rounded f32 operation, a
handful of them per score and weight, and what the chains of a stage or tile drop -- about 12 products of 2^-24 each on average --
come to 12 x 6e-8 = 7e-7 of the result's norm at worst, whatever the number of tokens."""
import math

import pytest
import torch

from tinycoder_inference_b200 import ops

pytestmark = pytest.mark.gpu
BOUND = 7e-7


def _far(q, k, v, out, pos):
    n, heads, hd = q.shape
    T, group = pos + n, heads // k.shape[1]
    mask = torch.arange(T, device="cuda")[None] > (pos + torch.arange(n, device="cuda"))[:, None]
    want = torch.empty((n, heads, hd), dtype=torch.float64, device="cuda")
    for h in range(heads):
        s = q[:, h].double() @ k[:T, h // group].double().T / math.sqrt(hd)
        want[:, h] = torch.softmax(s.masked_fill(mask, -math.inf), -1) @ v[:T, h // group].double()
    return float((out.double() - want).norm() / want.norm())


@pytest.mark.parametrize("dtype,nH,nKV,hd,rows,pos", [(torch.float32, 14, 2, 64, 512, 0), (torch.float32, 14, 2, 64, 512, 1000),
                                                      (torch.float32, 14, 2, 64, 200, 6000), (torch.float16, 14, 2, 64, 1500, 0),
                                                      (torch.float16, 14, 2, 64, 512, 1000), (torch.float16, 28, 4, 128, 512, 1000)])
def test_causal_rows(dtype, nH, nKV, hd, rows, pos):
    g = torch.Generator(device="cuda").manual_seed(rows + pos)
    q = torch.randn((rows, nH, hd), device="cuda", generator=g)
    k, v = (torch.randn((pos + rows, nKV, hd), device="cuda", generator=g).to(dtype) for _ in range(2))
    out = torch.empty_like(q)
    ops.prefill_kv(q, k, v, out, rows, nH, nKV, hd, pos)
    assert _far(q, k, v, out, pos) < BOUND


@pytest.mark.parametrize("nH,nKV,hd,pos", [(14, 2, 64, 16), (14, 2, 64, 20000), (28, 4, 128, 8191), (28, 4, 128, 40000)])
def test_fp16_decode(nH, nKV, hd, pos):
    """(with one running sum 7.9e-7 at 40000 rows, 4.2e-7 at 8191)"""
    far = []
    for seed in range(3):
        g = torch.Generator(device="cuda").manual_seed(seed)
        q = torch.randn((1, nH, hd), device="cuda", generator=g)
        k, v = (torch.randn((pos + 1, nKV, hd), device="cuda", generator=g).to(torch.float16) for _ in range(2))
        out = torch.empty_like(q)
        ops.decode_kv(q, k, v, out, ops.workspace(1, nH, hd, 256), 1, nH, nKV, hd, pos, 256)
        far.append(_far(q, k, v, out, pos))
    # a tile's chain is two products, not twelve: what is left is the rounding of scores, weights and sums
    assert sum(far) / 3 < 4e-7


@pytest.mark.parametrize("dtype,nH,nKV,hd,pos", [(torch.float16, 28, 4, 128, 9999), (torch.float16, 28, 4, 128, 16000), (torch.float16, 40, 8, 128, 4000),
                                                 (torch.float16, 40, 8, 128, 10000), (torch.float16, 14, 2, 64, 5000), (torch.float16, 8, 4, 64, 14000),
                                                 (torch.float32, 14, 2, 64, 3000), (torch.float32, 8, 4, 64, 5500)])
def test_decode_on_both_sides_of_the_merge(dtype, nH, nKV, hd, pos):
    """One token where a cluster of blocks folds a kv head's rows or a merge launch does.  (f32: up to sixteen tiles share a warp's sums, 1.3e-6 at
    most as measured; the bound is three times what a chain of 32 products drops, 32 x 6e-8.)"""
    g = torch.Generator(device="cuda").manual_seed(pos)
    q = torch.randn((1, nH, hd), device="cuda", generator=g)
    k, v = (torch.randn((pos + 1, nKV, hd), device="cuda", generator=g).to(dtype) for _ in range(2))
    out = torch.empty_like(q)
    ops.decode_kv(q, k, v, out, ops.workspace(1, nH, hd, 256), 1, nH, nKV, hd, pos, 256)
    assert _far(q, k, v, out, pos) < (BOUND if dtype == torch.float16 else 6e-6)


@pytest.mark.parametrize("dtype,nH,nKV,hd,pos", [(torch.float16, 40, 8, 128, 6500), (torch.float16, 28, 4, 128, 24000), (torch.float32, 8, 2, 128, 9000)])
def test_decode_without_partial_buffers(dtype, nH, nKV, hd, pos):
    """... is one cluster per kv head, in turns where they are not all resident, whatever the call with buffers takes.  Bounds as above; f32 rows
    of 16 blocks are up to 36 tiles a warp: 72 products in a sum."""
    g = torch.Generator(device="cuda").manual_seed(pos)
    q = torch.randn((1, nH, hd), device="cuda", generator=g)
    k, v = (torch.randn((pos + 1, nKV, hd), device="cuda", generator=g).to(dtype) for _ in range(2))
    out = torch.empty_like(q)
    ops.decode_kv(q, k, v, out, (None, None, None), 1, nH, nKV, hd, pos, 256)
    assert _far(q, k, v, out, pos) < (BOUND if dtype == torch.float16 else 72 * 6e-8 * 3)


@pytest.mark.parametrize("nH,nKV,pos", [(14, 2, 4000), (8, 4, 4000), (8, 4, 30000)])
def test_f32_decode_of_many_tiles_a_warp(nH, nKV, pos):
    """... at head_dim 64 is as near as 1500 rows, a tile a warp: what a warp adds up beyond a tile is f32.  (Means of eight inputs, which differ by some 3 %
    of each other; with one running sum 1.2 to 2.9 times as far.)"""
    def mean(pos):
        far = 0.0
        for seed in range(8):
            g = torch.Generator(device="cuda").manual_seed(seed)
            q = torch.randn((1, nH, 64), device="cuda", generator=g)
            k, v = (torch.randn((pos + 1, nKV, 64), device="cuda", generator=g) for _ in range(2))
            out = torch.empty_like(q)
            ops.decode_kv(q, k, v, out, ops.workspace(1, nH, 64, 256), 1, nH, nKV, 64, pos, 256)
            far += _far(q, k, v, out, pos) / 8
        return far

    assert mean(pos) < 1.15 * mean(1500)
