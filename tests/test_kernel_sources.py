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


def test_attributes_are_set_for_every_context():
    """A kernel's attributes belong to a device: set once per process, behind a
    static flag, they are missing on the next device that a context is made on.
    They are set at context creation only, and no launcher keeps a flag."""
    setters = set()
    for name in sorted(os.listdir(CSRC)):
        function = ""
        with open(os.path.join(CSRC, name)) as f:
            for line in f:
                assert "static bool" not in line, (name, line)
                start = re.match(r"[a-z][\w:<>*& ]* \**(\w+)\(", line)
                function = start.group(1) if start else function
                if "cudaFuncSetAttribute(" in line:
                    assert function.endswith("_set_attributes"), (name, function)
                    setters.add(function)
    with open(os.path.join(CSRC, "ctx.cu")) as f:
        create = f.read().split("int ngrav_gpu_create(")[1].split("\nvoid ngrav_gpu_destroy")[0]
    assert setters and all(fn + "();" in create for fn in setters), setters


@pytest.mark.parametrize("name,functions", [("engine.cuh", ["two_sum", "fast_two_sum", "df_offset", "df_add_prod"]),
                                            ("tree.cu", ["df_add"])])
def test_error_free_steps_name_their_roundings(name, functions):
    """A plain float sum may be fused with the product that an operand comes from,
    by the compiler's choice, and an error-free step is none any more."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    for fn in functions:
        bodies = re.findall(r"__forceinline__ void " + fn + r"\([^)]*\) \{(.*?)\n\}", text, re.S)
        assert len(bodies) == 1, fn
        assert not re.search(r" [-+*] ", bodies[0]), bodies[0]
