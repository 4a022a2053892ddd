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
