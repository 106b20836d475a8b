"""Truss decompositions with enough edges that the active list and the live lists are
compacted, and with enough live entries for the dense form: trussness from the
construction, and against k_truss, which peels without either."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G

pytestmark = pytest.mark.gpu


def edges_of(g):
    c = g.to_csr()
    rows = np.repeat(np.arange(g.num_nodes, dtype=np.uint32), np.diff(c.offsets.astype(np.int64)))
    return rows, c.targets


# Copies of cliques: K_n has trussness n and goes in one round of k = n + 1. Numbers of edges
# around the 131,072 from which lists are compacted, the halves going at different levels.
@pytest.mark.parametrize("sizes", [{2: 66_000, 3: 20_000, 5: 500}, {2: 65_000, 3: 1, 4: 900}, {3: 50_000, 10: 3000, 60: 80},
                                   {40: 200, 41: 100, 90: 60, 170: 25}, {700: 1, 300: 2, 30: 40, 2: 9}, {2: 300_000}])
def test_cliques(device, sizes):
    n, pairs, want = 0, [], []
    for size, copies in sizes.items():
        i, j = np.triu_indices(size, 1)
        base = n + size * np.arange(copies)[:, None]
        pairs.append(np.stack([(base + i).ravel(), (base + j).ravel()], 1))
        want.append(np.full(copies * len(i), size))
        n += size * copies
    pairs, want = np.concatenate(pairs), np.concatenate(want)
    name = np.random.default_rng(n).permutation(n + 5)  # five vertices without an edge
    a, b = name[pairs[:, 0]], name[pairs[:, 1]]
    g = G.GpuGraph.from_edge_pairs(np.stack([a, b], 1), n + 5, True, device)
    r = g.truss_decomposition()
    rows, cols = edges_of(g)
    key = rows.astype(np.int64) * (n + 5) + cols
    for x, y in ((a, b), (b, a)):
        assert np.array_equal(r["trussness"][np.searchsorted(key, x * (n + 5) + y)], want)
    # Every k up to the largest size ends with a round that removes nothing.
    assert (r["max_trussness"], r["rounds"]) == (max(sizes), max(sizes) - 2 + len(sizes))


@pytest.mark.parametrize("scale,edge_factor", [(13, 16), (15, 24), (17, 16)])
def test_trusses_of_the_decomposition(device, scale, edge_factor):
    g = G.GpuGraph.from_csr_arrays(G.generate_rmat(scale, edge_factor, 0.57, 0.19, 0.19, seed=scale), device)
    r = g.truss_decomposition()
    rows, cols = edges_of(g)
    once = rows < cols
    for k in (3, 4, 7, 12, r["max_trussness"] // 2, r["max_trussness"], r["max_trussness"] + 1):
        keep = once & (r["trussness"] >= k)
        assert np.array_equal(np.stack([rows[keep], cols[keep]], 1), g.k_truss_array(k)["edges"]), k
