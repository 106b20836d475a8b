"""Batched triangle counts in both forms: batches of sparse graphs without hubs, which
are counted over the DAG or over word lists, whichever was faster, and batches for
which the lists are shorter than the graphs, at the size from which both are tried.
Whole numbers: equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def noise(n, m, seed):
    c = G.from_edge_pairs(np.random.default_rng(seed).integers(0, n, size=(m, 2)), n, True)
    return c.offsets, c.targets


def grid(w, h):
    at = np.arange(w * h).reshape(h, w)
    c = G.from_edge_pairs(np.concatenate([np.stack([at[:, :-1].ravel(), at[:, 1:].ravel()], 1),
                                          np.stack([at[:-1].ravel(), at[1:].ravel()], 1),
                                          np.stack([at[:-1, :-1].ravel(), at[1:, 1:].ravel()], 1)]), w * h, True)
    return c.offsets, c.targets


@pytest.mark.parametrize("name", ["sparse", "small", "grids", "dense", "mixed", "empty"])
def test_both_forms(device, name):
    members = {"sparse": lambda: [noise(20_000 + 500 * i, 80_000, i) for i in range(5)],
               "small": lambda: [noise(8_000, 16_300, 1), noise(8_000, 16_500, 2)],  # about 65,536 entries
               "grids": lambda: [grid(60, 50), grid(41, 300), grid(200, 30), grid(7, 7)],
               "dense": lambda: [noise(300, 12_000, 3), noise(500, 40_000, 4), noise(64, 2000, 5)],
               "mixed": lambda: [noise(30_000, 200_000, 6), noise(400, 30_000, 7), grid(33, 3)],
               "empty": lambda: [(np.zeros(5, np.uint32), np.zeros(0, np.uint32))] * 3}[name]()
    b = G.GpuBatch.from_graphs(members, device)
    want = [O.triangle_count(o, t) for o, t in members]
    for _ in range(2):
        assert b.triangle_count()["total_triangles"].tolist() == want
    tuning = b.tuning()["triangle_buckets"]
    assert tuning.get("variant") == "word lists" or name in ("sparse", "small", "grids", "mixed")
