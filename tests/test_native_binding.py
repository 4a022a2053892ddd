"""The Python front's C++ binding: an argument that torch itself refuses is a Python exception, not the end of the process."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (a fake CUDA tensor has no address; asking it for one throws in C++)
FAKE = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from tinycoder_inference_b200 import capi, ops
with FakeTensorMode():
    f = torch.empty(8, 2, 128, device="cuda")
n = capi.native
"""
CALLS = {
    "wrapped call": "n.kv_append(f, f, f, f, 0, 8, 2, 128, 0, None, 8)",
    "attend": "n.attend(0, 0, f, f, f, f, 0, None, False)",
    "decode_i8_batch": "n.decode_i8_batch(f, *[None] * 15, *[1] * 8, 1.0, 0, 0, 0)",
}


@pytest.mark.parametrize("call", CALLS.values(), ids=CALLS.keys())
def test_a_cpp_exception_becomes_a_python_one(call):
    code = FAKE + f"try:\n    {call}\nexcept Exception as e:\n    print('raised', type(e).__name__)\n"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, f"exit code {r.returncode}: {r.stderr[-300:]}"
    assert r.stdout.startswith("raised"), r.stdout


@pytest.mark.gpu
def test_attend_refuses_a_q_without_dimensions():
    import torch

    from tinycoder_inference_b200 import ops

    s = ops.KvSession(8, 2, 128, 64, 1, mode="i8")
    kv = torch.zeros((1, 2, 128), device="cuda")
    with pytest.raises(IndexError):
        s.attend(0, torch.zeros((), device="cuda"), kv, kv, torch.zeros((1, 8, 128), device="cuda"), 0)


@pytest.mark.gpu
def test_other_threads_run_while_clear_waits_for_the_stream():
    import threading
    import time

    import torch

    from tinycoder_inference_b200 import ops

    s = ops.KvSession(8, 2, 128, 64, 1, mode="f32")
    s.clear()
    torch.cuda._sleep(1000)
    torch.cuda.synchronize()
    stamps, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            stamps.append(time.perf_counter())
            time.sleep(0.002)

    t = threading.Thread(target=tick)
    t.start()
    torch.cuda._sleep(800_000_000)      # about 0.4 s of the stream ahead of the synchronise in clear()
    a = time.perf_counter()
    s.clear()
    b = time.perf_counter()
    stop.set()
    t.join()
    assert b - a > 0.1, "the stream was not busy"
    inside = [x for x in stamps if a + 0.02 < x < b - 0.02]
    assert len(inside) > 5, f"{len(inside)} ticks of another thread in {b - a:.2f} s"
