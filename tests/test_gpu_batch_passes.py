"""The union passes of the batched BFS and PageRank where their parts meet: many
graphs in one 256-entry chunk, rows that cross several chunks, graphs without
vertices or entries, a last chunk of one entry, targets without entries of their
own, 1 to 32 sources, graphs that stop at different levels and iterations."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# FP32 ranks and contributions with FP64 sums: a rounding of at most 2^-24 of
# every rank per iteration, damped by 0.85 a step, stays below 2^-24 / 0.15 of a
# total rank of 1, twice (rank and contribution).
PPR_L1 = 2 * 2.0**-24 / 0.15


def csr(pairs, n, symmetric=True):
    c = G.from_edge_pairs(pairs, n, symmetric)
    return c.offsets, c.targets


def star(n):
    return csr(np.stack([np.zeros(n, np.int64), np.arange(1, n + 1)], 1), n + 1)


def path(n):
    return csr(np.stack([np.arange(n - 1), np.arange(1, n)], 1), n)


def noise(n, m, seed, symmetric=True):
    return csr(np.random.default_rng(seed).integers(0, n, size=(m, 2)), n, symmetric)


NO_VERTEX = (np.zeros(1, np.uint32), np.zeros(0, np.uint32))
NO_ENTRY = (np.zeros(6, np.uint32), np.zeros(0, np.uint32))


def graphs(name):
    if name == "tiny":
        return [path(2 + i % 5) for i in range(97)] + [NO_VERTEX, NO_ENTRY, path(3), NO_VERTEX]
    if name == "stars":  # the hub rows cross chunks; one ends on a chunk's last entry
        return [star(n) for n in (127, 128, 255, 256, 1023, 5000)] + [NO_VERTEX]
    if name == "one_entry_over":  # 257 entries in all
        return [star(128), (np.array([0, 1], np.uint32), np.array([0], np.uint32))]
    if name == "levels":  # paths stop late, the others early
        return [path(300), noise(500, 3000, 1), path(41), NO_ENTRY, noise(3001, 30000, 2), star(700)]
    return [noise(211, 900, 3, False), path(7), noise(64, 80, 4, False)]  # directed: targets without entries


@pytest.mark.parametrize("name", ["tiny", "stars", "one_entry_over", "levels", "directed"])
@pytest.mark.parametrize("per_graph", [1, 32])
def test_union_passes_match_oracle(device, name, per_graph):
    members = graphs(name)
    live = [m for m in members if len(m[0]) > 1]
    b = G.GpuBatch.from_graphs(live if per_graph == 32 else [m for m in members if len(m[0]) > 1], device)
    if name in ("tiny", "stars") and per_graph == 1:
        # Graphs without vertices only take part where no source is needed of them.
        assert G.GpuBatch.from_graphs(members, device).triangle_count()["total_triangles"].sum() == \
            b.triangle_count()["total_triangles"].sum()
    rng = np.random.default_rng(per_graph)
    sources = np.array([rng.integers(0, len(o) - 1, per_graph) for o, _ in live], dtype=np.uint32)
    seeds = np.array([rng.integers(0, len(o) - 1, min(per_graph, 3)) for o, _ in live], dtype=np.uint32)
    b.set_bfs_sources(sources)
    b.set_pagerank_seeds(seeds, 0.85, 60, 1e-5)
    b.capture()
    b.replay()
    r = b.results()
    direct = b.bfs()
    assert np.array_equal(r["distances"], direct["distances"])
    vb = b.vertex_base
    for g, (o, t) in enumerate(live):
        for k in range(per_graph):
            if name == "directed":
                # A level pulls over the lists: the search runs on the transpose.
                n = len(o) - 1
                src = np.repeat(np.arange(n), np.diff(o.astype(np.int64)))
                c = G.from_edge_pairs(np.stack([t.astype(np.int64), src], 1), n, False)
                ref = O.bfs(c.offsets, c.targets, int(sources[g, k]))
            else:
                ref = O.bfs(o, t, int(sources[g, k]))
            assert np.array_equal(r["distances"][k, vb[g]:vb[g + 1]], ref["distances"]), (g, k)
            assert r["reachable"][g, k] == ref["reachable"] and r["max_depth"][g, k] == ref["max_depth"], (g, k)
        n_it = int(r["iterations"][g])
        ref = O.pagerank(o, t, 0.85, n_it, 0.0, tele=O.seed_vector(len(o) - 1, seeds[g]))
        assert np.abs(r["ranks"][vb[g]:vb[g + 1]].astype(np.float64) - ref["ranks"]).sum() <= PPR_L1, g
        assert bool(r["converged"][g]) == (n_it < 60) or n_it == 60
