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
        want[:, h] = p @ v[:, kv].double().nan_to_num(0.0, 0.0, 0.0)  # (for rows that do not see what is not finite)
    assert ops.device_status() == 0
    return out, want


def _far(out, want):
    """The worst row's distance, relative to its norm."""
    return float(((out.double() - want).norm(dim=-1) / want.norm(dim=-1)).max())


@pytest.mark.parametrize("scale", [20, 28, 40, 80])
@pytest.mark.parametrize("which", ["q", "k"])
@pytest.mark.parametrize("S,nH,nKV,hd,pos", SIZES)
def test_a_large_row_of_q_or_k_leaves_its_neighbours_alone(which, scale, S, nH, nKV, hd, pos):
    """Row 33 times 2^scale: the other rows of q, or the rows in front of it, which do not see it."""
    q, k, v = _inputs(S, nH, nKV, hd, pos)
    (q if which == "q" else k[pos:])[33] *= 2.0 ** scale
    out, want = _run(q, k, v, pos)
    rest = [r for r in range(S) if r != 33] if which == "q" else list(range(33))
    assert _far(out[rest], want[rest]) < FAR


@pytest.mark.parametrize("size", [1e5, 1e8, 1e10, 1e20, 1e30])
@pytest.mark.parametrize("which", ["q", "k", "v", "v zeros"])
@pytest.mark.parametrize("S,nH,nKV,hd,pos", SIZES)
def test_one_large_dim_leaves_the_others_alone(which, size, S, nH, nKV, hd, pos):
    """A dim of every third row times `size`: the other dims of V, and scores in which that dim meets zeros.  "v zeros": these rows have nothing
    in their other dims, so that their weight, which outdoes all others, is no measure of those."""
    q, k, v = _inputs(S, nH, nKV, hd, pos)
    {"q": q, "k": k, "v": v, "v zeros": v}[which][::3, :, 5] *= size
    rest = [d for d in range(hd) if d != 5]
    if which == "q":
        k[..., 5] = 0.0
    elif which == "k":
        q[..., 5] = 0.0
    elif which == "v zeros":
        v[::3, :, rest] = 0.0
    out, want = _run(q, k, v, pos)
    some = slice(1 if which == "v zeros" and pos == 0 else 0, None)  # (row 0 sees nothing but zeros there)
    assert _far(out[some][..., rest], want[some][..., rest]) < FAR
    assert float((out - want)[..., 5].norm() / want[..., 5].norm()) < FAR


@pytest.mark.parametrize("size", [1e5, 1e8, 1e15, 1e30])
@pytest.mark.parametrize("S,nH,nKV,hd,pos", SIZES)
def test_large_rows_with_zeros_leave_the_other_dims_alone(size, S, nH, nKV, hd, pos):
    """Sixteen rows in a row of V with one dim other than 0, and that large: their weight says nothing about the other dims."""
    q, k, v = _inputs(S, nH, nKV, hd, pos)
    rest = [d for d in range(hd) if d != 5]
    v[pos + 16:pos + 32, :, rest] = 0.0
    v[pos + 16:pos + 32, :, 5] *= size
    out, want = _run(q, k, v, pos)
    assert _far(out[..., rest], want[..., rest]) < FAR


@pytest.mark.parametrize("what", [math.inf, -math.inf, math.nan])
@pytest.mark.parametrize("S,nH,nKV,hd,pos", SIZES)
def test_rows_ahead_of_one_that_is_not_finite_do_not_see_it(what, S, nH, nKV, hd, pos):
    q, k, v = _inputs(S, nH, nKV, hd, pos)
    v[pos + 33, :, 7] = what
    k[pos + 40] = what
    q[20] = what
    out, want = _run(q, k, v, pos)
    rest = [r for r in range(33) if r != 20]
    assert _far(out[rest], want[rest]) < FAR
    assert not torch.isfinite(out[20]).any() and not torch.isfinite(out[33:, :, 7]).any() and torch.isnan(out[40:]).any(-1).all()


@pytest.mark.parametrize("scale", [20, 28, 40, 100])
@pytest.mark.parametrize("S,nH,nKV,hd,pos", SIZES)
def test_a_large_row_of_v_weighs_what_its_probability_is(scale, S, nH, nKV, hd, pos):
    """Row 34 times 2^scale: rows that do not see it, and rows that do with a score far below the others'."""
    q, k, v = _inputs(S, nH, nKV, hd, pos)
    v[pos + 34] *= 2.0 ** scale
    out, want = _run(q, k, v, pos)
    assert _far(out[:34], want[:34]) < FAR
    # a dim of its own makes the score of row 34 lower by scale + 45 powers of two
    q[..., 0], k[..., 0] = 1.0, 0.0
    k[pos + 34, :, 0] = -(scale + 45.0) * math.log(2.0) * math.sqrt(hd)
    out, want = _run(q, k, v, pos)
    assert _far(out, want) < FAR


@pytest.mark.parametrize("past", [0, 5, 1000])
@pytest.mark.parametrize("S,nH,nKV,hd,rows", [(64, 40, 4, 64, 150), (64, 48, 8, 128, 77), (64, 64, 4, 256, 65)])
def test_a_device_position_past_the_store_attends_the_rows_there_are(past, S, nH, nKV, hd, rows):
    """The last stage is filled up with rows that nobody sees, also where the position on the device says that somebody does."""
    q, k, v = _inputs(S, nH, nKV, hd, rows - S)
    out = torch.full_like(q, float("nan"))
    at = torch.tensor([rows + past], dtype=torch.int32, device="cuda")
    ops.prefill_kv(q, k, v, out, S, nH, nKV, hd, 0, dev_pos=at)
    for h in range(nH):
        kv = h * nKV // nH
        want = torch.softmax(q[:, h].double() @ k[:, kv].double().T / math.sqrt(hd), -1) @ v[:, kv].double()
        assert _far(out[:, h], want) < FAR
