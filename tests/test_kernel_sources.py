"""Rules that the kernels' sources have to keep and that no run can show to hold: read here as text, without a GPU."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nvfp4_cutlass_b200", "csrc")
KERNELS = sorted(os.path.basename(f) for f in glob.glob(os.path.join(CSRC, "*.cu")))


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def enclosing(text, at):
    """Headers of the blocks around position `at`, and the names of the calls whose argument lists are open there."""
    blocks, calls, header = [], [], 0
    for i, c in enumerate(text[:at]):
        if c == "{":
            blocks.append(text[header:i])
            header = i + 1
        elif c == "}":
            blocks.pop()
            header = i + 1
        elif c == ";":
            header = i + 1
        elif c == "(":
            calls.append(re.search(r"[\w:]*$", text[:i]).group(0))
        elif c == ")":
            calls.pop()
    return blocks, calls


@pytest.mark.parametrize("name", KERNELS)
def test_a_warp_waits_as_one(name):
    """A bounded wait is made by one thread, or the warp votes on its outcome: lanes that leave a poll at different times
    must not reach a warp-wide instruction apart, and none may give up alone."""
    text = source(name)
    for m in re.finditer(r"ptx::mbar_wait\w*", text):
        blocks, calls = enclosing(text, m.start())
        by_one = any(re.search(r"\b(lane|threadIdx\.x) == 0\b", b) for b in blocks) or \
            "threadIdx.x == 0 &&" in text[text.rfind(";", 0, m.start()):m.start()]
        assert by_one or "ptx::all_lanes" in calls, f"{name}:{text.count(chr(10), 0, m.start()) + 1}"


def test_warp_wide_instructions_start_converged():
    """Allocation, release and the cluster barrier follow roles that one lane runs alone."""
    text = source("ptx.cuh")
    for mnemonic in ("tcgen05.alloc", "tcgen05.dealloc", "barrier.cluster.arrive"):
        places = [m.start() for m in re.finditer(re.escape(mnemonic), text)]
        assert places
        for at in places:
            assert "__syncwarp();" in text[text.rfind("{", 0, text.rfind("asm", 0, at)):at], mnemonic
