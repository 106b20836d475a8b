"""The passes' chunk lists: large graphs that stop one after the other until a deep
one is left, so that the list of the chunks at work is made anew several times, with
the graphs in any order. Distances are whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

PPR_L1 = 2 * 2.0**-24 / 0.15  # two FP32 roundings of a rank of 1 per iteration, damped by 0.85 a step


def csr(pairs, n):
    c = G.from_edge_pairs(np.asarray(pairs), n, True)
    return c.offsets, c.targets


def noise(n, m, seed):
    return csr(np.random.default_rng(seed).integers(0, n, size=(m, 2)), n)


def ladder(n, rungs, seed):
    """A path of n vertices with `rungs` shortcuts of up to nine: about n / 5 levels."""
    rng = np.random.default_rng(seed)
    a = rng.integers(0, n - 10, rungs)
    return csr(np.concatenate([np.stack([np.arange(n - 1), np.arange(1, n)], 1),
                               np.stack([a, a + rng.integers(2, 10, rungs)], 1)]), n)


@pytest.mark.parametrize("order", [0, 1])
def test_graphs_that_stop_one_after_the_other(device, order):
    # 5.9 M entries, 23,000 chunks: more than two a warp of a full grid.
    graphs = [noise(200_000, 1_300_000, 1), noise(100_000, 800_000, 2), ladder(60_000, 400_000, 3),
              ladder(20_000, 60_000, 4), noise(30_000, 400_000, 5), ladder(30_000, 9_000, 6), noise(500, 3000, 7)]
    if order:
        graphs = graphs[::-1]
    assert sum(len(t) for _, t in graphs) > 2 * 256 * 148 * 5 * 8
    b = G.GpuBatch.from_graphs(graphs, device)
    src = np.array([[0, len(o) // 2] for o, _ in graphs], dtype=np.uint32)
    b.set_bfs_sources(src)
    b.set_pagerank_seeds(src, 0.85, 80, 1e-6)
    vb = b.vertex_base
    for _ in range(2):
        r, p = b.bfs(), b.personalized_pagerank()
        for g, (o, t) in enumerate(graphs):
            for k in range(2):
                ref = O.bfs(o, t, int(src[g, k]))
                assert np.array_equal(r["distances"][k, vb[g]:vb[g + 1]], ref["distances"]), (g, k)
                assert (r["reachable"][g, k], r["max_depth"][g, k]) == (ref["reachable"], ref["max_depth"]), (g, k)
            n_it = int(p["iterations"][g])
            tele = O.seed_vector(len(o) - 1, src[g])
            ref = O.pagerank(o, t, 0.85, n_it, 0.0, tele=tele)["ranks"]
            assert np.abs(p["ranks"][vb[g]:vb[g + 1]].astype(np.float64) - ref).sum() <= PPR_L1, g
            assert abs(n_it - O.pagerank(o, t, 0.85, 80, 1e-6, tele=tele)["iterations"]) <= 1, g
    assert len(set(p["iterations"].tolist())) > 2
