"""Causal f32 rows in blocks of 32 whose numbers are of very different size: what is large in one place takes nothing from what
does not depend on it.  Against a 64-bit evaluation."""
import math

import pytest
import torch

from tinycoder_inference_b200 import ops

pytestmark = pytest.mark.gpu

# Every factor is held to 22 bits: a product is off by 2^-22 of itself at most, a score of N(0, 1) rows -- hd of them, times 1 / sqrt(hd) -- by
# 1.2 x 2^-22 = 2.9e-7 on average, and the worst of some ten thousand by five times that.  The weights of a row move by as much, and their
# sum with them: twice that of the row's norm.
FAR = 3e-6
SIZES = [(64, 40, 4, 64, 0), (64, 48, 8, 128, 0), (64, 64, 4, 256, 0), (70, 40, 2, 64, 130)]


def _inputs(S, nH, nKV, hd, pos):
    g = torch.Generator(device="cuda").manual_seed(S + hd + pos)
    q = torch.randn((S, nH, hd), device="cuda", generator=g)
    k, v = (torch.randn((pos + S, nKV, hd), device="cuda", generator=g) for _ in range(2))
    return q, k, v


def _run(q, k, v, pos):
    S, nH, hd = q.shape
    out = torch.full_like(q, float("nan"))
    ops.prefill_kv(q, k, v, out, S, nH, k.shape[1], hd, pos)
    mask = torch.arange(pos + S, device="cuda")[None] > (pos + torch.arange(S, device="cuda"))[:, None]
    want = torch.empty((S, nH, hd), dtype=torch.float64, device="cuda")
    for h in range(nH):
        kv = h * k.shape[1] // nH
        p = torch.softmax((q[:, h].double() @ k[:, kv].double().T / math.sqrt(hd)).masked_fill(mask, -math.inf), -1)
        want[:, h] = p @ v[:, kv].double()
    assert ops.device_status() == 0
    return out, want


def _far(out, want):
    """The worst row's distance, relative to its norm."""
    return float(((out.double() - want).norm(dim=-1) / want.norm(dim=-1)).max())


@pytest.mark.parametrize("scale", [20, 28, 40, 100])
@pytest.mark.parametrize("S,nH,nKV,hd,pos", SIZES)
def test_a_large_row_of_v_weighs_what_its_probability_is(scale, S, nH, nKV, hd, pos):
    """Row 34 times 2^scale: rows that do not see it, and one that does with a score far below the others'."""
    q, k, v = _inputs(S, nH, nKV, hd, pos)
    v[pos + 34] *= 2.0 ** scale
    out, want = _run(q, k, v, pos)
    assert _far(out[:34], want[:34]) < FAR
    # a dim of its own makes the score of row 34 lower by scale + 45 powers of two
    q[..., 0], k[..., 0] = 1.0, 0.0
    k[pos + 34, :, 0] = -(scale + 45.0) * math.log(2.0) * math.sqrt(hd)
    out, want = _run(q, k, v, pos)
    assert _far(out[:35], want[:35]) < FAR
