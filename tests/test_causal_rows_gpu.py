"""Causal rows in blocks of 32 (many rows and heads: fewer rows take the 8-row form), at the edges of their row tiles and of
their stages of 128 / 64 / 32 tokens, with host and device positions."""
import math

import numpy as np
import pytest
import torch

import oracle
from tinycoder_inference_b200 import ops
from tests.util import assert_close, dev, host

pytestmark = pytest.mark.gpu

# Products of hi + lo pairs keep each factor to 2^-21: a score of N(0, 1) rows moves by 3 * 2^-21 * 0.64 sqrt(hd) <= 1.5e-5,
# an output by twice that times the largest |v| (4.5).
ATOL = 1.4e-4


SIZES = [(9, 128, 8, 64, 5), (33, 64, 8, 64, 95), (129, 40, 2, 64, 130), (200, 14, 2, 64, 0), (32, 80, 8, 128, 32),
         (65, 48, 8, 128, 0), (129, 28, 4, 128, 40), (16, 160, 16, 256, 0), (47, 64, 4, 256, 16), (97, 32, 2, 256, 0)]


@pytest.mark.parametrize("S,nH,nKV,hd,pos,half", [(*c, half) for c in SIZES for half in (False, True)
                                                  if not (half and c[3] == 256)])  # (no fp16 store at head_dim 256)
def test_blocks_of_32_rows(S, nH, nKV, hd, pos, half):
    r = np.random.default_rng(S + nH + pos)
    rows = pos + S
    q = r.standard_normal((S, nH, hd), dtype=np.float32)
    k, v = (r.standard_normal((rows + 3, nKV, hd), dtype=np.float32) for _ in range(2))
    if half:
        k, v = k.astype(np.float16), v.astype(np.float16)
    k[rows:] = np.nan  # rows behind the last one attended may hold anything
    v[rows:] = np.nan
    want = oracle.attention_kv(q, k, v, S, nH, nKV, hd, pos, 1.0 / math.sqrt(hd))
    kd, vd, at = dev(k), dev(v), torch.tensor([pos], dtype=torch.int32, device="cuda")
    for where in ({}, {"dev_pos": at}):
        out = torch.full((S + 1, nH, hd), float("nan"), device="cuda")
        ops.prefill_kv(dev(q), kd, vd, out[:S], S, nH, nKV, hd, 0 if where else pos, **where)
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        assert_close(host(out[:S]), want, rtol=0.0, atol=ATOL, what=f"{S} rows, {where}")
        assert torch.isnan(out[S]).all()  # a ragged last block writes its own rows only


def _rows(r, S, nH, nKV, hd, pos, qScale, kScale, vScale, kSpread=12, vSpread=16):
    q = r.standard_normal((S, nH, hd)) * 2.0 ** qScale
    k = r.standard_normal((pos + S, nKV, hd)) * 2.0 ** (kScale - r.integers(0, kSpread, (pos + S, 1, 1)))
    v = r.standard_normal((pos + S, nKV, hd)) * 2.0 ** (vScale - r.integers(0, vSpread, (pos + S, 1, 1)))
    return (x.astype(np.float32) for x in (q, k, v))


def _want(q, k, v, pos):
    """The same in 64 bits, [rows][heads][hd]."""
    S, nH, hd = q.shape
    out = np.empty(q.shape)
    mask = np.arange(k.shape[0])[None] > pos + np.arange(S)[:, None]
    for h in range(nH):
        s = q[:, h].astype(np.float64) @ k[:, h // (nH // k.shape[1])].astype(np.float64).T / math.sqrt(hd)
        s[mask] = -np.inf
        p = np.exp(s - s.max(1, keepdims=True))
        out[:, h] = (p / p.sum(1, keepdims=True)) @ v[:, h // (nH // k.shape[1])].astype(np.float64)
    return out


@pytest.mark.parametrize("kSpread,vSpread", [(12, 16), (60, 80)])
@pytest.mark.parametrize("qScale,kScale,vScale", [(0, 0, 0), (40, -40, 60), (-60, 62, -90)])
@pytest.mark.parametrize("S,nH,nKV,hd,pos", [(33, 64, 8, 64, 95), (200, 14, 2, 64, 1), (65, 48, 8, 128, 63), (47, 64, 4, 256, 17)])
def test_rows_of_any_magnitude(S, nH, nKV, hd, pos, qScale, kScale, vScale, kSpread, vSpread):
    """The f32 form takes its operands apart relative to the largest element of some rows: rows of K and V up to 2^11 and 2^15 apart, which the pairs hold,
    and up to 2^59 and 2^79, which they do not, next to one another and as a whole.  Bound, against the norm of a row's result: that of N(0, 1) rows
    (tests/test_exact_range_gpu.py), times what the scores are larger by."""
    q, k, v = _rows(np.random.default_rng(S + pos), S, nH, nKV, hd, pos, qScale, kScale, vScale, kSpread, vSpread)
    out = torch.full((S, nH, hd), float("nan"), device="cuda")
    ops.prefill_kv(dev(q), dev(k), dev(v), out, S, nH, nKV, hd, pos)
    want = _want(q, k, v, pos)
    err = np.linalg.norm(host(out).astype(np.float64) - want, axis=2) / np.linalg.norm(want, axis=2)
    assert err.max() < 3e-6 * 2.0 ** (qScale + kScale)


@pytest.mark.parametrize("hd,nH,nKV", [(64, 64, 8), (128, 48, 8), (256, 64, 4)])
def test_values_that_are_not_finite_stay_in_their_dims(hd, nH, nKV):
    """An infinity in a V row reaches its own dim only, and a K row with NaN the rows that see it.  (Rows ahead of them: tests/test_exact_range_gpu.py.)"""
    S, pos = 70, 30
    q, k, v = _rows(np.random.default_rng(hd), S, nH, nKV, hd, pos, 0, 0, 0)
    want = _want(q, k, v, pos)
    bad = v.copy()
    bad[pos + 1, :, 5] = np.inf
    bad[pos + 2, :, 7] = np.nan
    out = torch.full((S, nH, hd), float("nan"), device="cuda")
    ops.prefill_kv(dev(q), dev(k), dev(bad), out, S, nH, nKV, hd, pos)
    rest = [d for d in range(hd) if d not in (5, 7)]
    got = host(out)
    assert_close(got[..., rest], want[..., rest], rtol=0.0, atol=ATOL)
    assert not np.isfinite(got[2:, :, [5, 7]]).any()
    k[pos + S - 1] = np.nan  # the last row sees it, nobody else
    ops.prefill_kv(dev(q), dev(k), dev(v), out, S, nH, nKV, hd, pos)
    got = host(out)
    assert_close(got[:-1], want[:-1], rtol=0.0, atol=ATOL)
    assert np.isnan(got[-1]).all()
