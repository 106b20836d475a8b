"""Device CSR builds at the edges of the radix sort's and the builder's tiles.

The sort takes 2,048-key tiles, as many per block as make one wave of blocks, and
8-bit digits over the target and source bits as one number, so digits straddle
the two words for most id widths. Pairs and sorted keys are read in 2,048-key
tiles. Every CSR equals the oracle's.
"""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(device, pairs, n, symmetric):
    g = G.GpuGraph.from_edge_pairs(pairs, n, symmetric, device)
    o, t = O.from_edge_pairs(pairs, n, symmetric)[:2]
    csr = g.to_csr()
    assert np.array_equal(csr.offsets, o) and np.array_equal(csr.targets, t)
    return g


def draw(rng, m, n):
    """Random pairs, self-loops, repeats and both directions among them."""
    p = rng.integers(0, n, size=(m, 2), dtype=np.uint32)
    if m > 3:
        p[m // 2] = p[0]
        p[m // 3] = p[0][::-1]
        p[m - 1] = (n - 1, n - 1)
    return p


@pytest.mark.parametrize("m", [0, 1, 2, 31, 255, 2047, 2048, 2049, 4096, 65537, 592 * 2048 - 1, 592 * 2048,
                               592 * 2048 + 1, 3 * 592 * 2048 + 77])
@pytest.mark.parametrize("symmetric", [False, True])
def test_sizes(device, m, symmetric):
    rng = np.random.default_rng(m + symmetric)
    check(device, draw(rng, m, 70000), 70000, symmetric)


@pytest.mark.parametrize("bits", [0, 1, 3, 4, 5, 7, 8, 9, 11, 12, 13, 15, 16, 17, 20, 21, 23, 24])
def test_id_widths(device, bits):
    n = 1 << bits
    rng = np.random.default_rng(bits)
    for count in {n, n - 1, n + 1} - {0}:
        g = check(device, draw(rng, 9001, count), count, True)
        check(device, draw(rng, 9001, count), count, False)
    # The directed plan sorts by target alone; the in-lists keep their order.
    r = g.pagerank_directed(0.85, 3, 0.0)
    csr = g.to_csr()
    s = G.GpuGraph.from_csr(csr.offsets, csr.targets, device).pagerank_array(0.85, 3, 0.0)
    assert np.allclose(r["ranks"], s["ranks"], rtol=1e-5, atol=1e-9)  # symmetric: pull over itself


def test_one_source(device):
    """Every key in one bucket of the source digits, then of the target digits."""
    a = np.arange(200_001, dtype=np.uint32)
    check(device, np.stack([np.full_like(a, 5), a], 1), 200_001, False)
    check(device, np.stack([a, np.full_like(a, 5)], 1), 200_001, False)
    check(device, np.stack([np.full_like(a, 5), a[::-1]], 1), 200_001, True)


def test_oriented(device):
    rng = np.random.default_rng(3)
    p = draw(rng, 100_003, 5000)
    g = G.GpuGraph.from_edge_pairs_oriented(p, 5000, device)
    host = G.from_edge_pairs_oriented(p, 5000)
    csr = g.to_csr()
    assert np.array_equal(csr.offsets, host.offsets) and np.array_equal(csr.targets, host.targets)
