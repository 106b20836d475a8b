"""Triangle counts over word lists at the sizes where the lists change form: rows
of 32 / 33 and 128 / 129 neighbours, owners around the warp kernel's limits (96
words, 512 neighbours), rows of several items, ranks beyond one bitmap window.
Whole numbers: equal to the oracle's, to a closed form, or to the count over the
oriented CSR (triangle_trace, which runs every variant of it)."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def clique(n, first=0):
    i, j = np.triu_indices(n, 1)
    return np.stack([i + first, j + first], 1)


def pairs_of(name):
    rng = np.random.default_rng(len(name))
    if name.startswith("clique"):
        n = int(name[6:])
        return clique(n), n
    if name.startswith("wheel"):  # a hub over a ring: rim rows of 3, a hub row of n
        n = int(name[5:])
        rim = np.arange(1, n + 1)
        return np.concatenate([np.stack([np.zeros(n, np.int64), rim], 1), np.stack([rim, np.roll(rim, 1)], 1)]), n + 1
    if name == "mixed":  # many sizes side by side, with bridges and isolated vertices
        sizes, at, out = [2, 3, 31, 32, 33, 34, 96, 97, 98, 127, 128, 129, 130], 5, []
        for k in sizes:
            out.append(clique(k, at))
            at += k
        return np.concatenate(out + [np.array([[5, at - 1], [6, 7], [40, 41]])]), at + 3
    if name == "loops":
        p = rng.integers(0, 300, size=(6000, 2))
        return np.concatenate([p, np.stack([np.arange(300), np.arange(300)], 1)]), 300
    n, m = (int(x) for x in name[4:].split("x"))  # rand
    return rng.integers(0, n, size=(m, 2)), n


@pytest.mark.parametrize("name", ["clique3", "clique33", "clique130", "clique600", "wheel511", "wheel513", "wheel5000",
                                  "mixed", "loops", "rand50x100", "rand700x60000", "rand3000x300000",
                                  "rand40000x400000"])
def test_word_lists_match_oracle(device, name):
    pairs, n = pairs_of(name)
    c = G.from_edge_pairs(pairs, n, True)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    expect = O.triangle_count(c.offsets, c.targets)
    assert g.triangle_count()["total_triangles"] == expect
    b = G.GpuBatch.from_graphs([(c.offsets, c.targets), (c.offsets, c.targets)], device)
    assert b.triangle_count()["total_triangles"].tolist() == [expect, expect]


def test_ranks_beyond_one_window(device):
    # A ring lattice: all of one degree class, ranks are ids, 140 neighbours each.
    n, half = 270001, 70
    g = G.GpuGraph.generate_watts_strogatz(device, n, 2 * half, 0.0)
    assert g.triangle_count()["total_triangles"] == n * half * (half - 1) // 2
    # Owners of about 110 words (the CTA kernel) with ranks in a second window.
    g = G.GpuGraph.generate_erdos_renyi(device, 300007, 110 * 300007, seed=5)
    assert g.triangle_count()["total_triangles"] == g.triangle_trace()["total_triangles"]
