"""Searches of graphs that come and go: the buffers of each come from memory in
which the searches of the graphs before have left their own items, and each
graph's searches are numbered from the start. The levels have 512 to 16,384
frontier edges, which a group of blocks runs by handing tagged items over.
Whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def grid(w, h, symmetric=True):
    at = np.arange(w * h).reshape(h, w)
    p = np.concatenate([np.stack([at[:, :-1].ravel(), at[:, 1:].ravel()], 1),
                        np.stack([at[:-1].ravel(), at[1:].ravel()], 1)])
    c = G.from_edge_pairs(p[np.random.default_rng(w + h).random(len(p)) >= 0.03], w * h, symmetric)
    return c.offsets, c.targets


def layers(width, count):
    """Layers of `width` vertices, each joined to three of the next: frontiers of one size."""
    at = np.arange(width * count).reshape(count, width)
    rng = np.random.default_rng(width)
    p = np.concatenate([np.stack([at[:-1].ravel(), np.roll(at[1:], s, axis=1).ravel()], 1)
                        for s in rng.integers(0, width, 3)] + [np.stack([np.zeros(width, np.int64), at[0]], 1)])
    c = G.from_edge_pairs(p, width * count, True)
    return c.offsets, c.targets


def test_graphs_searched_and_dropped_in_turn(device):
    shapes = [grid(900, 900), grid(211, 157), layers(2500, 40), grid(131, 600), layers(600, 9), grid(400, 64, False),
              grid(640, 640), layers(130, 30)]
    runs = []
    for o, t in shapes:
        for s in (0, (len(o) - 1) // 2):
            runs.append((o, t, s, O.bfs(o, t, s)))
    order = np.random.default_rng(1)
    for turn in range(160):
        # A large graph, then a smaller one, now and then searched again.
        o, t, s, ref = runs[int(order.integers(0, len(runs))) if turn % 2 else 2 * (turn % 3) % len(runs)]
        g = G.GpuGraph.from_csr(o, t, device)
        for _ in range(1 + turn % 3 // 2):
            r = g.bfs_array(s)
            assert np.array_equal(r["distances"], ref["distances"]), (turn, len(o) - 1, s)
            assert (r["reachable"], r["max_depth"]) == (ref["reachable"], ref["max_depth"])
        del g
