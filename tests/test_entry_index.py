"""Entry index arithmetic of the kernels (csrc/entry_index.h) for lists that end
within a few entries of 2^32, where a rounded-up position would wrap: compiled
for the host and compared with unbounded integers.

The walks are those of the kernels: a lane's or a warp's loop over an item (the
BFS stretches), the warp's loop over a row (the triangle owners), the cut of an
item into pieces for several warps, and the items of a list."""
from __future__ import annotations

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import PKG

HARNESS = r"""
#include "entry_index.h"
#include <vector>
using namespace gcu;
extern "C" {
uint32_t t_count(uint32_t d, uint32_t size) { return range_count(d, size); }
void t_range(uint32_t s, uint32_t d, uint32_t size, uint32_t c, uint32_t* out) {
    out[0] = range_begin(s, size, c);
    out[1] = range_end(s, d, size, c);
}
void t_piece(uint32_t x, uint32_t y, uint32_t part, uint32_t piece, uint32_t* out) {
    take_piece(x, y, part, piece);
    out[0] = x;
    out[1] = y;
}
// The entries that `lanes` lanes take, `unroll` at a time, in a walk of [s, e); -1: too many steps.
int64_t t_walk(uint32_t s, uint32_t e, uint32_t lanes, uint32_t unroll, uint32_t* out, int64_t room) {
    int64_t n = 0, steps = 0;
    bool bad = false;
    walk_entries(s, e, lanes * unroll, [&](uint32_t o) {
        if (++steps > room) { bad = true; return; }
        for (uint32_t lane = 0; lane < lanes; ++lane) {
            const uint32_t at = entry_or_end(s, e, o, lane);
            for (uint32_t u = 0; u < unroll; ++u)
                if (at < e && e - at > u * lanes) {
                    if (n < room) out[n] = at + u * lanes;
                    ++n;
                }
        }
    });
    return bad ? -1 : n;
}
}
"""

TOP = (1 << 32) - 1  # the largest number of entries


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("entry_index")
    src, so = d / "t.cpp", d / "t.so"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(PKG, "csrc"), str(src), "-o",
                    str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.t_count.restype = C.c_uint32
    lib.t_walk.restype = C.c_int64
    return lib


def pair(f, *args):
    out = (C.c_uint32 * 2)()
    f(*[C.c_uint32(a) for a in args], out)
    return out[0], out[1]


@pytest.mark.parametrize("d", [0, 1, 1023, 1024, 1025, 4097, TOP - 1024, TOP - 1, TOP])
@pytest.mark.parametrize("size", [256, 1024])
def test_ranges_of_a_list(lib, d, size):
    n = lib.t_count(C.c_uint32(d), C.c_uint32(size))
    assert n == -(-d // size)
    for s in {0, TOP - d}:
        for c in {0, 1, n // 2, n - 2, n - 1} & set(range(n)):
            assert pair(lib.t_range, s, d, size, c) == (s + c * size, s + min(d, (c + 1) * size))


@pytest.mark.parametrize("length", [1, 2, 31, 33, 511, 1023, 1024])
@pytest.mark.parametrize("end", [2000, TOP - 1024, TOP - 1, TOP])
def test_pieces_cover_an_item(lib, length, end):
    x, y = end - length, end
    for parts in (1, 2, 3, 7, 16):
        for piece in {-(-length // parts), length // parts + 1}:
            got = [pair(lib.t_piece, x, y, p, piece) for p in range(parts)]
            assert [i for a, b in got for i in range(a, b)] == list(range(x, y))
            assert all(x <= a <= b <= y for a, b in got)


@pytest.mark.parametrize("length", [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 1000, 1024])
@pytest.mark.parametrize("end", [1024, TOP - 64, TOP - 31, TOP - 1, TOP])
def test_walks_take_each_entry_once(lib, length, end):
    s = end - length
    for lanes in (1, 4, 16, 32):
        for unroll in (1, 2):
            out = np.zeros(4096, dtype=np.uint32)
            n = lib.t_walk(C.c_uint32(s), C.c_uint32(end), C.c_uint32(lanes), C.c_uint32(unroll),
                           out.ctypes.data_as(C.POINTER(C.c_uint32)), C.c_int64(4096))
            assert n == length
            assert np.array_equal(np.sort(out[:n]).astype(np.int64), np.arange(s, end))
