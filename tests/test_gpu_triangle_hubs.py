"""Word lists of hubs, whose rows are read many entries at a time or, where few
vertices rank below them, searched for those: rows around the limits, hubs joined to
one another or not, self-loops at them, and vertices of one neighbour, which are in
no triangle. Counts and edges are whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def graph(hubs, leaves, joined, noise, seed):
    """`hubs` hubs over the same `leaves` vertices (joined: to one another too), a self-loop at
    every other one, `noise` random pairs, and vertices of one neighbour behind."""
    rng = np.random.default_rng(seed)
    n = hubs + leaves
    p = [np.stack([np.full(leaves, h), np.arange(hubs, n)], 1) for h in range(hubs)]
    if joined:
        p.append(np.stack(np.triu_indices(hubs, 1), 1))
    p.append(np.stack([np.arange(0, hubs, 2)] * 2, 1))
    p.append(rng.integers(0, n, size=(noise, 2)))
    tail = np.arange(n, n + 501)
    p.append(np.stack([tail, rng.integers(0, n, 501)], 1))
    p.append(np.array([[n + 501, n + 502], [n + 503, n + 503]]))
    return G.from_edge_pairs(np.concatenate(p), n + 504, True)


@pytest.mark.parametrize("hubs,leaves,joined,noise", [(1, 50_000, False, 0), (1, 129, False, 40), (2, 50_000, True, 500),
                                                      (8, 15_000, True, 3000), (40, 1279, True, 200),
                                                      (40, 1281, False, 200), (100, 3300, True, 5000),
                                                      (200, 2500, False, 8000), (5, 20_000, True, 30_000)])
def test_hubs(device, hubs, leaves, joined, noise):
    c = graph(hubs, leaves, joined, noise, hubs + leaves)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    assert g.triangle_count()["total_triangles"] == O.triangle_count(c.offsets, c.targets)
    b = G.GpuBatch.from_graphs([(c.offsets, c.targets), (c.offsets, c.targets)], device)
    assert len(set(b.triangle_count()["total_triangles"].tolist()) | {O.triangle_count(c.offsets, c.targets)}) == 1
    for k in (3, 5):
        r, ref = g.k_truss_array(k), O.k_truss(c.offsets, c.targets, k)
        assert np.array_equal(r["edges"], ref["edges"]) and r["iterations"] == ref["iterations"], k


def test_hub_beyond_one_bitmap(device):
    """More vertices than the supports' bitmap holds: the hub's list is made in two windows. The
    hub makes a triangle with every pair of leaves that are joined."""
    n, m = 1_800_000, 30_000
    ends = np.random.default_rng(3).permutation(np.arange(1, n))[:2 * m].reshape(m, 2)  # a matching
    p = np.concatenate([np.stack([np.zeros(n - 1, np.int64), np.arange(1, n)], 1), ends])
    c = G.from_edge_pairs(p, n, True)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    assert g.triangle_count()["total_triangles"] == m
    r = g.k_truss_array(3)
    want = np.concatenate([np.stack([np.zeros(2 * m, np.int64), np.sort(ends.ravel())], 1), np.sort(ends, axis=1)])
    want = want[np.lexsort((want[:, 1], want[:, 0]))]
    assert np.array_equal(r["edges"], want) and r["iterations"] == 2
