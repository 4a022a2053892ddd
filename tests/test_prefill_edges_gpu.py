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
