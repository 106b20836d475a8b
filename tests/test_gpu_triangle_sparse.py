"""Triangles, edge supports and batches of sparse graphs, where most word lists have
one word: lists of one neighbour own no edge, and an edge between lists of one word
is the higher rank's. Forests, short cycles, small cliques and sparse random graphs
with ids in any order, so that ids and ranks disagree; equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def pairs_of(name, n):
    rng = np.random.default_rng(n)
    i = np.arange(1, n)
    if name == "binary tree":
        p = np.stack([i, (i - 1) // 2], 1)
    elif name == "random tree":
        p = np.stack([i, (rng.random(n - 1) * i).astype(np.int64)], 1)
    elif name == "triangles":  # a cactus of them
        k = np.arange(1, n - 1, 2)
        a = (rng.random(len(k)) * k).astype(np.int64)
        p = np.concatenate([np.stack([k, k + 1], 1), np.stack([a, k], 1), np.stack([a, k + 1], 1)])
    elif name == "cliques":  # of 3 to 7, some joined
        sizes = rng.integers(3, 8, n // 7)
        at = np.concatenate([[0], np.cumsum(sizes)[:-1]])
        p = np.concatenate([np.stack(np.triu_indices(s, 1), 1) + b for s, b in zip(sizes, at)]
                           + [rng.integers(0, sizes.sum(), size=(n // 20, 2))])
    else:  # a random graph of `name` edges per vertex
        p = rng.integers(0, n, size=(int(float(name) * n), 2))
    return rng.permutation(n)[p]


@pytest.mark.parametrize("n", [3, 40, 1000, 70_001])
@pytest.mark.parametrize("name", ["binary tree", "random tree", "triangles", "cliques", "0.7", "1.5", "4"])
def test_sparse_graphs(device, name, n):
    if n < 7 and name in ("cliques", "0.7"):
        return
    c = G.from_edge_pairs(pairs_of(name, n), n, True)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    expect = O.triangle_count(c.offsets, c.targets)
    assert g.triangle_count()["total_triangles"] == expect
    if name.endswith("tree"):
        assert expect == 0
    b = G.GpuBatch.from_graphs([(c.offsets, c.targets)] * 3, device)
    assert b.triangle_count()["total_triangles"].tolist() == [expect] * 3
    for k in (3, 4):
        r, ref = g.k_truss_array(k), O.k_truss(c.offsets, c.targets, k)
        assert np.array_equal(r["edges"], ref["edges"]) and r["iterations"] == ref["iterations"]
