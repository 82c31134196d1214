"""Instructions that a whole warp has to execute together (``.sync.aligned``) follow a point where it is known to be
together: threads that took different ways through a branch or a loop come back together only there.  Host test of the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "torkit3d_b200", "csrc")
ASM = re.compile(r'asm\s+volatile\s*\(\s*"([^"]*)"')


def _unconverged(text):
    """Statements with .sync.aligned that are not preceded by __syncwarp(), __syncthreads() or another one of them."""
    text = re.sub(r"//[^\n]*", "", text)
    found = []
    together = -1  # where the last such statement, or a barrier, ended
    for m in ASM.finditer(text):
        if ".sync.aligned" not in m.group(1):
            continue
        before = text[:m.start()].rstrip()
        if not (before.endswith(("__syncwarp();", "__syncthreads();")) or len(before) == together):
            found.append(m.group(1))
        depth, i = 0, text.index("(", m.start())
        quoted = False
        while True:  # the statement's end
            c = text[i]
            quoted ^= c == '"'
            depth += (c == "(") - (c == ")") if not quoted else 0
            i += 1
            if depth == 0:
                break
        together = text.index(";", i) + 1
    return found


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh"))))
def test_warps_are_together_at_aligned_instructions(name):
    with open(os.path.join(CSRC, name)) as f:
        assert _unconverged(f.read()) == []


def test_the_check_sees_a_missing_barrier():
    good = '__syncwarp();\n  asm volatile("a.sync.aligned;" ::"r"(f(x)) : "memory");\n asm volatile("b.sync.aligned;");'
    assert _unconverged(good) == []
    assert _unconverged("if (lane == 0) work();\n" + good[len("__syncwarp();"):]) == ["a.sync.aligned;"]
    assert _unconverged(good.replace(' asm volatile("b', ' if (c) d(); asm volatile("b')) == ["b.sync.aligned;"]
