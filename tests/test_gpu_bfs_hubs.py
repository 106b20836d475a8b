"""BFS of directed CSRs whose frontiers hold long lists among short ones: the items of
a long list are consecutive in the queue and are spread over the warps. Lists of one
to several items (1,024 entries each) at their edges, few and many leaves, leaves
before and after the hubs; equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def hubs_and_leaves(degrees, leaves, back, seed):
    """Vertex 0 leads to every hub and leaf, a hub to `degree` vertices of a second
    layer, a leaf to `back` of them."""
    rng = np.random.default_rng(seed)
    h, n2 = len(degrees), max(degrees)
    second = 1 + h + leaves
    ids = rng.permutation(np.arange(1, second))  # hubs and leaves in any order
    pairs = [np.stack([np.zeros(h + leaves, np.int64), ids], 1)]
    for k, d in enumerate(degrees):
        pairs.append(np.stack([np.full(d, ids[k]), second + rng.permutation(n2)[:d]], 1))
    for _ in range(back):
        pairs.append(np.stack([ids[h:], second + rng.integers(0, n2, leaves)], 1))
    pairs.append(np.stack([second + np.arange(n2), rng.integers(0, second, n2)], 1))
    return G.from_edge_pairs(np.concatenate(pairs), second + n2, False)


@pytest.mark.parametrize("degrees, leaves, back", [
    ((1023, 1024, 1025, 2048, 2049), 20_000, 1),
    ((300_000,), 3, 2), ((300_000, 299_000, 5000), 200_000, 3), ((9000,) * 40, 31, 2), ((200_000,) * 3, 5000, 4),
    ((70_000, 20_000, 10), 60_000, 1)])
def test_long_lists_among_short_ones(device, degrees, leaves, back):
    c = hubs_and_leaves(degrees, leaves, back, sum(degrees) + leaves)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    for s in (0, 1, len(degrees) + leaves, len(c.offsets) - 2):
        r, ref = g.bfs_array(s), O.bfs(c.offsets, c.targets, s)
        assert np.array_equal(r["distances"], ref["distances"])
        assert (r["reachable"], r["max_depth"]) == (ref["reachable"], ref["max_depth"])


@pytest.mark.parametrize("hubs, leaves", [(1, 40_000), (3, 50_000), (16, 30_000)])
def test_half_of_a_symmetric_graph(device, hubs, leaves):
    """Hubs with the same leaves, each entry kept with odds of a half."""
    p = np.concatenate([np.stack([np.full(leaves, k), np.arange(hubs, hubs + leaves)], 1) for k in range(hubs)])
    p = np.concatenate([p, p[:, ::-1]])
    p = p[np.random.default_rng(hubs).random(len(p)) < 0.5]
    c = G.from_edge_pairs(p, hubs + leaves, False)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    for s in (0, hubs - 1, hubs, hubs + leaves - 1):
        r, ref = g.bfs_array(s), O.bfs(c.offsets, c.targets, s)
        assert np.array_equal(r["distances"], ref["distances"])
        assert (r["reachable"], r["max_depth"]) == (ref["reachable"], ref["max_depth"])
