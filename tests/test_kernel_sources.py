"""Properties of the device code that a run cannot show: it may work by the
compiler's choice of the day, and a failing case could hang a GPU.  They are
read off the sources."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opengl-physics_gb300", "csrc")


def statements(name):
    """The file's statements in order, comments gone, white space folded."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    text = re.sub(r"//[^\n]*", "", text)
    return [" ".join(s.split()) for s in re.split(r";(?=\s)(?!\\n)|(?<=[{}])\s", text) if s.strip()]


@pytest.mark.parametrize("name", ["tree.cu", "tc.cuh"])
def test_aligned_instructions_follow_a_reconvergence(name):
    """An .aligned instruction needs all threads of its warp at it together, so
    one comes directly after __syncwarp() (or after another of its kind)."""
    before, found = "", 0
    for s in statements(name):
        if "asm volatile" in s and ".aligned" in s:
            found += 1
            assert before.endswith("__syncwarp()") or ".aligned" in before, s
        before = s
    assert found
