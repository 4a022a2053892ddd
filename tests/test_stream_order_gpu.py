"""A decode call that reads old rows ahead of its dependency wait (TC_DECODE_PDL) behind calls that wrote those rows: what
it reads early is what the stream's order says.  Every round writes other rows, so a row read too early shows."""
import pytest
import torch

from tinycoder_inference_b200 import ops

pytestmark = pytest.mark.gpu
NH, NKV, HD, ROUNDS = 28, 4, 128, 24


def _pool(rows):
    k8 = torch.zeros((rows, NKV, HD), dtype=torch.int8, device="cuda")
    return [k8, torch.zeros_like(k8), torch.ones((rows, NKV), device="cuda"), torch.ones((rows, NKV), device="cuda")]


def _early(q, pool, out, ws, length, prefetch_rows, new=None):
    ops.decode_i8_batch(q, *pool, out, ws, None, 1, NH, NKV, HD, length, 64, rows_per_seq=length, pdl=True,
                        prefetch_rows=prefetch_rows, append=new)


def _rounds(pos, write, early):
    """Per round: write(rows of the round), then the early reader -- once in one go, once with a wait in between."""
    g = torch.Generator(device="cuda").manual_seed(pos)
    rn = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    ws = ops.workspace(1, NH, HD, 64)
    got, want = [], []
    data = [(rn(pos + 1, NKV, HD), rn(pos + 1, NKV, HD), rn(1, NH, HD)) for _ in range(2)]
    for wait, outs in ((False, got), (True, want)):
        for i in range(ROUNDS):
            out = torch.zeros((1, NH, HD), device="cuda")
            write(*data[i % 2])
            if wait:
                torch.cuda.synchronize()
            early(*data[i % 2], out, ws)
            outs.append(out)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    assert not torch.equal(want[0], want[1])
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), f"round {i} read rows before they were written"


# one block's rows, a cluster's, blocks and a merge; behind a second call that runs in a few blocks
@pytest.mark.parametrize("between", [False, True])
@pytest.mark.parametrize("pos", [100, 3000, 20000])
def test_rows_of_the_quantise_launch(pos, between):
    pool, other = _pool(pos + 16), _pool(512)
    out2, ws2, q2 = torch.zeros((1, NH, HD), device="cuda"), ops.workspace(1, NH, HD, 8), torch.zeros((1, NH, HD), device="cuda")

    def write(k, v, q):
        ops.kv_quantize_i8(k, v, *pool, pos, NKV, HD)
        if between:
            ops.decode_i8(q2, *other, out2, ws2, NH, NKV, HD, 400, 8)

    def early(k, v, q, out, ws):
        _early(q, pool, out, ws, pos + 1, pos, (k[pos:], v[pos:]))

    _rounds(pos, write, early)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("pos", [127, 3000])
def test_the_row_of_a_session_step(pos, captured):
    s = ops.KvSession(NH, NKV, HD, pos + 1, 1, mode="i8")
    pool = [t[0] for t in (s.k8, s.v8, s.ks, s.vs)]
    for t, x in zip(pool, _pool(pos + 17)):
        t.copy_(x)
    step, at = torch.zeros((1, NH, HD), device="cuda"), torch.tensor([pos], dtype=torch.int32, device="cuda")

    def write(k, v, q):
        # (a row far from the others: it carries the whole output)
        s.attend(0, q, 50.0 * k[pos:], 50.0 * v[pos:], step, pos, dev_pos=at if captured else None, graph_capture=captured)

    def early(k, v, q, out, ws):
        _early(q, pool, out, ws, pos + 1, pos + 1)

    _rounds(pos, write, early)
