"""No kernel counts a 32-bit position up to the end of a list or of a graph's
vertices in steps of more than one: where that end is within a step of 2^32 the
position wraps below it, and the walk does not end. Walks count offsets from the
beginning instead, or in 64 bits."""
from __future__ import annotations

import os
import re

from conftest import PKG

CSRC = os.path.join(PKG, "csrc")
END = r"(?:e|le|ae|be|xe|ye|row_end|\w+\.(?:v_end|e_end))"
STEPPED = re.compile(r"for \((?:uint32_t|unsigned) (\w+) = [^;]*;[^;]*\b\1 < " + END + r"\b(?!\s*[-\[(.])[^;]*; \1 \+= [^)]*\)")


def test_the_check_finds_a_stepped_walk():
    assert STEPPED.search("for (uint32_t j = s + lane; j < e; j += 32)")
    assert STEPPED.search("for (uint32_t v = g.v_begin + threadIdx.x; v < g.v_end; v += kThreads) x = 0;")
    assert not STEPPED.search("for (uint64_t j = s + lane; j < e; j += 32)")
    assert not STEPPED.search("for (uint32_t o = lane; o < e - s; o += 32)")
    assert not STEPPED.search("for (uint32_t j = s; j < e; ++j)")


def test_walks_do_not_step_past_an_end():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                assert [m.group(0) for m in STEPPED.finditer(f.read())] == [], name
