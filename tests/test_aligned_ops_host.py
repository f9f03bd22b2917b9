"""Warp-collective tensor-memory instructions (tcgen05.*.sync.aligned) need all 32 lanes together.
Lanes take different branches between them (stores past the volume's end or the layer's channels,
elected producer lanes), and nothing but an explicit barrier makes a warp converge again.  So each
function that issues such an instruction converges the warp itself, in the statement before it
(no GPU: the sources are read)."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ettention_b200", "csrc")


def _statements(body):
    """The statements of a function body without strings' line breaks and comments."""
    body = re.sub(r"//[^\n]*", "", body)
    return [" ".join(s.split()) for s in body.split(";\n")]


def test_every_aligned_tensor_memory_instruction_follows_a_warp_barrier():
    seen = 0
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        src = open(path).read()
        for m in re.finditer(r"asm volatile\(\s*\"tcgen05\.[\w:.]*\.sync\.aligned", src):
            start = src.rfind("\n__device__", 0, m.start())
            before = _statements(src[start:m.start()])
            # the barrier itself, or another aligned instruction right after one
            prev = [s for s in before[1 if len(before) > 1 else 0:] if s] or [""]
            held = before[0].endswith("{ __syncwarp()") and all("sync.aligned" in s for s in prev if s)
            assert held, src[start:m.end()]
            seen += 1
    assert seen >= 5  # alloc, relinquish, dealloc, ld, wait::ld


def test_warp_wide_waits_have_one_outcome():
    """A warp whose lanes go on to a tensor-memory read waits with mbar_wait_warp: a plain
    mbar_wait may give up in some lanes only."""
    src = open(os.path.join(CSRC, "learned.cuh")).read()
    assert "__all_sync(0xffffffffu, mbar_wait(" in src
    waits = re.findall(r"const bool got = (\w+)\(", src)
    assert waits and set(waits) == {"mbar_wait_warp"}
