"""The batched BFS and PageRank where a graph changes sides: the small graphs, a block
each, and the large ones, all together pass by pass. Sizes at the limits between
them and between the block sizes, many and few of a kind, rows longer than a lane
takes, and graphs whose entries begin and end anywhere in the large ones' chunks."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# Two FP32 roundings of a total rank of 1 per iteration, damped by 0.85 a step.
PPR_L1 = 2 * 2.0**-24 / 0.15


def csr(pairs, n, symmetric=True):
    c = G.from_edge_pairs(np.asarray(pairs), n, symmetric)
    return c.offsets, c.targets


def noise(n, m, seed, symmetric=True):
    return csr(np.random.default_rng(seed).integers(0, n, size=(m, 2)), n, symmetric)


def path(n):
    return csr(np.stack([np.arange(n - 1), np.arange(1, n)], 1), n)


def star(n):
    return csr(np.stack([np.zeros(n, np.int64), np.arange(1, n + 1)], 1), n + 1)


def sized(entries, n=4000):
    """A graph of exactly `entries` entries: a path, and pairs across it."""
    rng = np.random.default_rng(entries)
    want = entries // 2
    keys = {(i, i + 1) for i in range(min(n - 1, want))}
    while len(keys) < want:
        a, b = (int(x) for x in rng.integers(0, n, 2))
        if a != b:
            keys.add((min(a, b), max(a, b)))
    loops = [(0, 0)] if entries % 2 else []
    o, t = csr(list(keys) + loops, n)
    assert len(t) == entries
    return o, t


def members(name):
    if name == "alone":  # without larger ones 65,536 entries and vertices are small
        return [sized(65536), sized(65535, 9000), csr([(0, 1), (1, 2)], 65536), noise(2000, 20000, 8)]
    if name == "entries":  # beside larger graphs 32,768 entries are the most of a small one
        return [sized(32767), sized(32768), sized(32769), noise(300, 900, 1), sized(65537), sized(33003)]
    if name == "vertices":  # as are 32,768 vertices (of 65,537 here)
        return [csr([(0, 1), (1, 2)], n) for n in (32767, 32768, 32769)] + [csr([(5, 6)], 40001), path(3), csr([(0, 65536)], 65537)]
    if name == "classes":  # 512 and 2,048 vertices, more than two graphs an SM of each class
        return [noise(40 + i % 473, 700, i) for i in range(310)] + \
            [noise(513 + 5 * i, 1500, i) for i in range(307)] + [noise(n, 5000, n) for n in (512, 513, 2048, 2049)]
    if name == "rows":  # 31 entries a lane's, 32 a warp's; hubs on either side
        return [star(30), star(31), star(32), star(63), star(64), star(65), star(16000), star(20000), star(33000)]
    return [noise(211, 900, 3, False), noise(9000, 40000, 5, False), noise(64, 80, 4, False),
            noise(5000, 33000, 6, False), csr([], 3), csr([], 33000)]  # directed


@pytest.mark.parametrize("name", ["alone", "entries", "vertices", "classes", "rows", "directed"])
@pytest.mark.parametrize("per_graph", [1, 7])
def test_small_and_large_graphs(device, name, per_graph):
    graphs = members(name)
    if name == "classes" and per_graph > 1:
        graphs = graphs[::40]
    b = G.GpuBatch.from_graphs(graphs, device)
    rng = np.random.default_rng(per_graph)
    src = np.array([rng.integers(0, len(o) - 1, per_graph) for o, _ in graphs], dtype=np.uint32)
    b.set_bfs_sources(src)
    b.set_pagerank_seeds(src, 0.85, 40, 1e-5)
    r = b.bfs()
    p = b.personalized_pagerank()
    b.capture()
    b.replay()
    again = b.results()
    assert np.array_equal(r["distances"], again["distances"]) and np.array_equal(p["ranks"], again["ranks"])
    assert np.array_equal(p["iterations"], again["iterations"])
    vb = b.vertex_base
    for g, (o, t) in enumerate(graphs):
        n = len(o) - 1
        if name == "directed":  # a level pulls over the lists: the search runs on the transpose
            rows = np.repeat(np.arange(n), np.diff(o.astype(np.int64)))
            so, st = csr(np.stack([t.astype(np.int64), rows], 1), n, False)
        else:
            so, st = o, t
        for k in range(per_graph):
            ref = O.bfs(so, st, int(src[g, k]))
            assert np.array_equal(r["distances"][k, vb[g]:vb[g + 1]], ref["distances"]), (g, k)
            assert (r["reachable"][g, k], r["max_depth"][g, k]) == (ref["reachable"], ref["max_depth"]), (g, k)
        n_it = int(p["iterations"][g])
        ref = O.pagerank(o, t, 0.85, n_it, 0.0, tele=O.seed_vector(n, src[g]))["ranks"]
        mass = max(1.0, ref.sum())  # a directed graph pulled over its own lists may gain some
        assert np.abs(p["ranks"][vb[g]:vb[g + 1]].astype(np.float64) - ref).sum() <= PPR_L1 * mass, g
        want = O.pagerank(o, t, 0.85, 40, 1e-5, tele=O.seed_vector(n, src[g]))
        assert abs(n_it - want["iterations"]) <= 1, g
