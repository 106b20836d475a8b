"""Truss decomposition of hubs with long lists: the removed edges between them are
walks that all warps share. Trussness and rounds follow from the construction."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G

pytestmark = pytest.mark.gpu


def hubs(count, leaves, triangles):
    """`count` hubs in a ring, each neighbouring pair with one vertex joined to both, so that
    a ring edge is in one triangle; each hub's leaves in cliques of six, joined to it (every
    such edge in five triangles); and triangles of their own."""
    e, n = [], count
    for h in range(count):
        lv = n + h * leaves + np.arange(leaves)
        e.append((np.full(leaves, h), lv))
        c = lv.reshape(-1, 6)
        e += [(c[:, a], c[:, b]) for a in range(6) for b in range(a + 1, 6)]
    n += count * leaves
    cliques = len(e)
    h, nxt, x = np.arange(count), (np.arange(count) + 1) % count, n + np.arange(count)
    e += [(h, nxt), (h, x), (nxt, x)]
    t = n + count + np.arange(3 * triangles).reshape(-1, 3)
    e += [(t[:, 0], t[:, 1]), (t[:, 1], t[:, 2]), (t[:, 0], t[:, 2])]
    n += count + 3 * triangles
    expected = np.concatenate([np.full(len(a), 7 if i < cliques else 3) for i, (a, _) in enumerate(e)])
    pairs = np.concatenate([np.stack(p, 1) for p in e])
    return pairs, n, expected


# With many edges removed beside them a walk of 8,193 entries is long; alone, up to 16
# warps share an edge first.
@pytest.mark.parametrize("count,leaves,triangles", [(4, 8190, 4000), (4, 8196, 4000), (5, 60_000, 4000),
                                                    (3, 150_000, 0), (3, 120_000, 1), (40, 9000, 3000)])
def test_edges_between_hubs(device, count, leaves, triangles):
    pairs, n, expected = hubs(count, leaves, triangles)
    c = G.from_edge_pairs(pairs, n, True)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    r = g.truss_decomposition()
    rows = np.repeat(np.arange(n, dtype=np.int64), np.diff(c.offsets.astype(np.int64)))
    key = rows * n + c.targets
    at = np.searchsorted(key, np.minimum(pairs[:, 0], pairs[:, 1]) * n + np.maximum(pairs[:, 0], pairs[:, 1]))
    assert np.array_equal(r["trussness"][at], expected)
    back = np.searchsorted(key, np.maximum(pairs[:, 0], pairs[:, 1]) * n + np.minimum(pairs[:, 0], pairs[:, 1]))
    assert np.array_equal(r["trussness"][back], expected)
    # k = 4 removes in one round and ends in another; k = 3 and 5 to 7 remove nothing, k = 8 all
    # that is left. A ring of three is a triangle itself: its edges go a round after their others.
    assert (r["max_trussness"], r["rounds"]) == (7, 8 if count == 3 else 7)
