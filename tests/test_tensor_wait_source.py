"""Asynchronous tensor-memory loads in the sources are complete when their
registers can be read.

tcgen05.ld returns before its destination registers hold the data, and only a
tcgen05.wait::ld behind it makes them readable.  Two asm statements order the
instructions but not the plain arithmetic on the registers between or after them,
which the compiler may move; a load and its wait in one statement cannot be
separated.  Read from the source, since a compiled program that happens to be
scheduled well shows nothing.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flint_b200", "csrc")


def asm_statements(text):
    """The instruction text of every asm statement (adjacent literals joined)."""
    text = re.sub(r"//[^\n]*", "", text)
    out = []
    for m in re.finditer(r"\basm\s+(?:volatile\s*)?\(", text):
        lit, pos = [], m.end()
        while True:
            s = re.match(r'\s*"((?:[^"\\]|\\.)*)"', text[pos:])
            if not s:
                break
            lit.append(s.group(1))
            pos += s.end()
        out.append("".join(lit))
    return out


def files():
    return sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.inc")))


@pytest.mark.parametrize("path", files(), ids=os.path.basename)
def test_tensor_loads_end_with_their_wait(path):
    for s in asm_statements(open(path).read()):
        if "tcgen05.ld" in s:
            assert "tcgen05.wait::ld" in s[s.index("tcgen05.ld"):], s[:80]


def test_the_row_pass_has_such_loads():
    text = "".join(open(p).read() for p in files())
    assert any("tcgen05.ld" in s for s in asm_statements(text))


@pytest.mark.parametrize("path", files(), ids=os.path.basename)
def test_warps_converge_after_a_polled_wait(path):
    """tcgen05's .sync.aligned instructions need the whole warp together; a loop
    of polls that each thread leaves by itself does not bring it there, so a
    warp-wide decision and a __syncwarp stand between the poll and what follows."""
    text = re.sub(r"//[^\n]*", "", open(path).read())
    for m in re.finditer(r"(?<!bool )\btc_mbar_wait\s*\(", text):
        line = text[text.rindex("\n", 0, m.start()):m.start()]
        assert re.search(r"__(all|any)_sync\s*\(\s*0xffffffffu\s*,\s*!?$", line), line
        rest = text[m.end():]
        assert "__syncwarp()" in rest[:rest.index("tc_fence_after()")]
