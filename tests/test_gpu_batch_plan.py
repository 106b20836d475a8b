"""The triangle plan of sparse batches at its limits: lists without owners (paths,
cycles), and degree buckets below, at and above the 65,536 vertices from which a
bucket's variant is not timed. Counts equal the oracle's, also by replay."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def csr(p, n):
    c = G.from_edge_pairs(p, n, True)
    return c.offsets, c.targets


def path(n, closed=False):
    i = np.arange(n - 1)
    p = np.stack([i, i + 1], 1)
    return csr(np.concatenate([p, [[n - 1, 0]]]) if closed else p, n)


def regular(n, half):
    """Every vertex joined to `half` others on, at distances that make triangles."""
    i = np.arange(n)
    return csr(np.concatenate([np.stack([i, (i + k) % n], 1) for k in range(1, half + 1)]), n)


@pytest.mark.parametrize("name", ["paths", "cycles", "path and clique", "65,535", "65,536", "buckets"])
def test_plans(device, name):
    rng = np.random.default_rng(len(name))
    members = {"paths": lambda: [path(20_001), path(16_384), path(3), path(2)],
               "cycles": lambda: [path(40_000, True), path(3, True), path(4, True)],
               "path and clique": lambda: [path(60_000), csr(np.stack(np.triu_indices(9, 1), 1), 9)],
               "65,535": lambda: [regular(65_535, 20)],
               "65,536": lambda: [regular(65_536, 20)],
               "buckets": lambda: [csr(rng.integers(0, 200_000, size=(5_000_000, 2)), 200_000),
                                   csr(rng.integers(0, 30_000, size=(60_000, 2)), 30_000)]}[name]()
    b = G.GpuBatch.from_graphs(members, device)
    want = [O.triangle_count(o, t) for o, t in members]
    assert b.triangle_count()["total_triangles"].tolist() == want
    zeros = np.zeros((len(members), 1), dtype=np.uint32)
    b.set_bfs_sources(zeros, keep_distances=False)
    b.set_pagerank_seeds(zeros, 0.85, 2, 0.0)
    b.capture()
    b.replay()
    assert b.results(distances=False)["total_triangles"].tolist() == want
