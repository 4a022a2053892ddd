"""Rules for the device code that reading decides, not a run (breaking one may hang a GPU)."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tinycoder_inference_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def test_asm_that_synchronises_is_volatile():
    """An asm statement that is not volatile is a function of its operands: the compiler may move it to where its result
    is used, say under a test of the lane, and a warp-wide operation is then run by part of the warp."""
    seen, bad = 0, []
    for name in SOURCES:
        for m in re.finditer(r"\basm\b(\s+volatile\b)?\s*\(((?:\s*\"(?:[^\"\\]|\\.)*\")+)", _code(name)):
            if re.search(r"\.sync\b|\bbar\.|\bbarrier\.|mbarrier\.|tcgen05\.|cp\.async|griddepcontrol", m.group(2)):
                seen += 1
                if not m.group(1):
                    bad.append((name, m.group(2).strip()))
    assert seen > 30 and bad == []


def test_tensor_memory_is_given_back_behind_the_warps_that_issue():
    """A wait that ran out in some warps must not free tensor memory that others still issue products into: in front of each
    deallocation stands a barrier of the block, or the one that the issuing warps arrive at when they are through."""
    found = 0
    for name in SOURCES:
        lines = _code(name).splitlines()
        for i, line in enumerate(lines):
            if "tmemDealloc(" not in line or "__device__" in line:
                continue
            found += 1
            before = "\n".join(x for x in lines[:i] if x.strip()).splitlines()[-5:]
            barrier = re.search(r"__syncthreads\(\)|namedBarSync\((kIssuedBar), ", "\n".join(before))
            assert barrier, (name, i + 1)
            if barrier.group(1):
                assert "namedBarArrive(kIssuedBar, " in "\n".join(lines[:i]), (name, i + 1)
    assert found >= 2
