"""The truss decomposition's loop kernel at the edges of its paths.

Its rounds, level skips and compactions run in one kernel; searched lists are
staged in shared memory up to 512 entries, or looked up in rows of bits where
those are dense enough, and a round of few edges shares each edge's walk among
warps. Every result is a whole number: trussness, the largest
and the round count equal the oracle's peeling of the same CSR.
"""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def to_csr(n: int, pairs: np.ndarray, loops=()) -> tuple[np.ndarray, np.ndarray]:
    both = np.concatenate([pairs, pairs[:, ::-1], np.array([[v, v] for v in loops], dtype=np.int64).reshape(-1, 2)])
    key = np.unique(both[:, 0] * n + both[:, 1])
    src, dst = key // n, key % n
    return np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint32), dst.astype(np.uint32)


def clique(first: int, size: int) -> np.ndarray:
    a, b = np.triu_indices(size, 1)
    return np.stack([a + first, b + first], axis=1)


def disjoint_cliques(sizes) -> tuple[int, np.ndarray]:
    starts = np.concatenate([[0], np.cumsum(sizes)])
    return int(starts[-1]), np.concatenate([clique(int(s), z) for s, z in zip(starts, sizes)])


def dense(n: int, p: float, seed: int) -> tuple[int, np.ndarray]:
    all_pairs = clique(0, n)
    return n, all_pairs[np.random.default_rng(seed).random(len(all_pairs)) < p]


def ladder(n: int) -> tuple[int, np.ndarray]:
    """A strip of triangles and its tail: rounds of a few edges, one after another."""
    i = np.arange(n - 2)
    return n, np.concatenate([np.stack([i, i + 1], 1), np.stack([i, i + 2], 1)])


def hubs(leaves: int) -> tuple[int, np.ndarray]:
    """Two hubs sharing every leaf (lists far beyond the stage), and a clique on the first leaves."""
    v = np.arange(2, leaves + 2)
    return leaves + 2, np.concatenate([[[0, 1]], np.stack([0 * v, v], 1), np.stack([0 * v + 1, v], 1), clique(2, 12)])


def fringed(n: int, core: int, seed: int) -> tuple[int, np.ndarray]:
    """A dense core and low-degree vertices across all ids: rows of bits in which
    short lists are looked up."""
    rng = np.random.default_rng(seed)
    members = rng.choice(n, size=core, replace=False)
    a, b = np.triu_indices(core, 1)
    keep = rng.random(len(a)) < 0.5
    fringe = np.stack([np.repeat(np.arange(n), 6), rng.choice(members, size=6 * n)], 1)
    p = np.sort(np.concatenate([np.stack([members[a[keep]], members[b[keep]]], 1), fringe]), axis=1)
    return n, np.unique(p[p[:, 0] != p[:, 1]], axis=0)


GRAPHS = {
    "stage-1": lambda: disjoint_cliques([512]),  # live lists of 511
    "stage": lambda: disjoint_cliques([513, 5]),
    "stage+1": lambda: disjoint_cliques([514, 4, 3]),
    "levels": lambda: disjoint_cliques([3, 3, 4, 9, 33, 34, 70, 2, 2]),
    "halves": lambda: disjoint_cliques([3] * 6000 + [6] * 700 + [14] * 60 + [40] * 4),  # a compaction per level
    "dense": lambda: dense(900, 0.62, 3),
    "rows-1": lambda: dense(1023, 0.1, 7),  # of bits: one word less than a warp's 32
    "rows": lambda: dense(1024, 0.1, 8),
    "rows+1": lambda: dense(1025, 0.1, 9),
    "fringe": lambda: fringed(4000, 600, 10),
    "wide fringe": lambda: fringed(20000, 1500, 11),
    "sparse": lambda: dense(3000, 0.02, 5),
    "ladder": lambda: ladder(301),
    "hubs": lambda: hubs(5000),
    "one edge": lambda: (2, np.array([[0, 1]])),
}


@pytest.mark.parametrize("name", list(GRAPHS))
def test_truss_loop(device, name):
    n, pairs = GRAPHS[name]()
    o, t = to_csr(n, pairs)
    r = G.GpuGraph.from_csr(o, t, device).truss_decomposition()
    ref = O.truss_decomposition_peel(o, t)
    assert np.array_equal(r["trussness"], ref["trussness"])
    assert r["max_trussness"] == ref["max_trussness"]
    assert r["rounds"] == ref["rounds"]
    # Self-loops change neither the trussness of the other entries nor get one.
    loops = list(range(0, n, 3))
    lo, lt = to_csr(n, pairs, loops)
    lr = G.GpuGraph.from_csr(lo, lt, device).truss_decomposition()
    row = np.repeat(np.arange(n, dtype=np.uint32), np.diff(lo))
    assert np.array_equal(lr["trussness"][row != lt], ref["trussness"])
    assert not lr["trussness"][row == lt].any()
