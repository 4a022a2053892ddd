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
