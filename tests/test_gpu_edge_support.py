"""Edge supports from full word lists, over every block size and table.

The bitmap of an owner's neighbours covers all vertices up to 1.7 M (blocks of
128 to 1024 threads by its size), several windows or a hash table beyond. The
graphs' hubs reach every part of the rank range, and close triangles with and
without each other; trussness and rounds, whole numbers that follow from the
supports, equal the oracle's peeling.
"""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def graph(n: int, hubs: list[int], seed: int) -> tuple[np.ndarray, np.ndarray]:
    """A strip of triangles over all vertices, and hubs of the given degrees."""
    rng = np.random.default_rng(seed)
    i = np.arange(n, dtype=np.int64)
    parts = [np.stack([i, (i + 1) % n], 1), np.stack([i, (i + 2) % n], 1)]
    for k, d in enumerate(hubs):
        others = rng.choice(n, size=min(d, n - 1), replace=False)
        hub = n // 3 + 7 * k
        parts.append(np.stack([np.full(len(others), hub), others], 1))
        some = rng.choice(others, size=(2 * len(others) // 3, 2))  # edges between the hub's neighbours
        parts.append(some)
    parts.append(n // 3 + 7 * rng.integers(0, len(hubs), size=(40, 2)))  # between hubs
    p = np.concatenate(parts)
    p = p[p[:, 0] != p[:, 1]]
    key = np.unique(np.concatenate([p[:, 0] * n + p[:, 1], p[:, 1] * n + p[:, 0]]))
    src, dst = key // n, key % n
    return np.concatenate([[0], np.cumsum(np.bincount(src, minlength=n))]).astype(np.uint32), dst.astype(np.uint32)


@pytest.mark.parametrize("n,hubs", [
    (37, [9, 30]),
    (1500, [64, 65, 128, 129, 700]),       # warp and block owners
    (131072, [40, 200, 5000, 30000]),      # the largest bitmap of 128 threads
    (131073, [40, 200, 5000, 30000]),
    (270336, [100, 3000, 60000]),          # of 256
    (270337, [100, 3000, 60000]),
    (540672, [100, 3000, 90000]),          # of 512
    (540673, [100, 3000, 90000]),
    (1703936, [64, 300, 1024, 50000]),     # one window of 1024 threads
    (1703937, [64, 300, 1023, 1024, 1025, 50000]),  # two, or a hash table
    (3500001, [300, 4000, 200000]),        # three
])
def test_edge_support(device, n, hubs):
    o, t = graph(n, hubs, n)
    r = G.GpuGraph.from_csr(o, t, device).truss_decomposition()
    ref = O.truss_decomposition_peel(o, t)
    assert np.array_equal(r["trussness"], ref["trussness"])
    assert r["max_trussness"] == ref["max_trussness"] and r["rounds"] == ref["rounds"]
