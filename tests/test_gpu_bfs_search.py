"""The one-launch BFS at the sizes where its parts meet: vertex counts off the
tile widths, hubs of many items, frontiers around the single-block limit, paths
longer than one single-block stretch, both pull forms, directed CSRs. Distances,
`reachable` and `max_depth` are whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def pairs_of(name):
    """(pairs, vertices, symmetric, sources)"""
    rng = np.random.default_rng(len(name))
    if name == "one_vertex":
        return np.zeros((0, 2), np.int64), 1, True, [0]
    if name.startswith("star"):  # one hub: leaves around the item size and the single-block limit
        n = int(name[4:])
        return np.stack([np.zeros(n, np.int64), np.arange(1, n + 1)], 1), n + 1, True, [0, n]
    if name == "two_hubs":  # a path into a hub whose leaves all reach a second hub
        n = 9000
        a = np.stack([np.full(n, 3), np.arange(5, n + 5)], 1)
        b = np.stack([np.arange(5, n + 5), np.full(n, 4)], 1)
        return np.concatenate([[[0, 1], [1, 2], [2, 3]], a, b]), n + 5, True, [0, 4, 5]
    if name == "path":  # more levels than one single-block stretch
        n = 40001
        return np.stack([np.arange(n - 1), np.arange(1, n)], 1), n, True, [0, n // 2]
    if name.startswith("grid"):
        w, h = (int(x) for x in name[4:].split("x"))
        at = np.arange(w * h).reshape(h, w)
        p = np.concatenate([np.stack([at[:, :-1].ravel(), at[:, 1:].ravel()], 1),
                            np.stack([at[:-1].ravel(), at[1:].ravel()], 1)])
        return p[rng.random(len(p)) >= 0.05], w * h, True, [0, w * h // 2 + w // 2]
    if name == "directed":
        return rng.integers(0, 20011, size=(120000, 2)), 20011, False, [1, 17, 20010]
    if name == "directed_grid":
        p, n, _, s = pairs_of("grid257x129")
        return p, n, False, s
    if name.startswith("random"):  # isolated vertices: the list form of the pull
        n = int(name[6:])
        return rng.integers(0, n // 2, size=(8 * n, 2)), n, True, [0, 1, n - 1]
    n = int(name[2:])  # er: no isolated vertex
    return np.concatenate([rng.integers(0, n, size=(6 * n, 2)), np.stack([np.arange(n - 1), np.arange(1, n)], 1)]), \
        n, True, [0, n - 1]


@pytest.mark.parametrize("name", ["one_vertex", "star255", "star256", "star257", "star8191", "star8193", "star70000",
                                  "two_hubs", "path", "grid31x33", "grid257x129", "grid700x601", "directed",
                                  "directed_grid", "random1000", "random65537", "er33", "er4097", "er65535"])
def test_one_launch_search_matches_oracle(device, name):
    pairs, n, symmetric, sources = pairs_of(name)
    c = G.from_edge_pairs(pairs, n, symmetric)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    for s in sources:
        ref = O.bfs(c.offsets, c.targets, int(s))
        for _ in range(2):  # a repeat finds the buffers as the last search left them
            r = g.bfs_array(int(s))
            assert np.array_equal(r["distances"], ref["distances"]), (name, s)
            assert (r["reachable"], r["max_depth"]) == (ref["reachable"], ref["max_depth"]), (name, s)
