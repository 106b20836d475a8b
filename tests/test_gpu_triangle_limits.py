"""Triangle counts and edge supports over word lists at the limits that decide who
counts an owner: a warp up to 128 neighbours in up to 64 words (32 words in a graph
below 524,288 vertices), a block beyond either. Equal to the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def owners_over_hubs(words, rows, n):
    """A circulant of 66 * 32 vertices of about 300 neighbours, which rank first and in
    order, and for each of `words` x `rows` an owner joined to that many of them in
    that many words."""
    hubs = 66 * 32
    at = np.arange(hubs)
    pairs = [np.stack([at, (at + k) % hubs], 1) for k in range(1, 151)]
    u = hubs
    rng = np.random.default_rng(n)
    for w in words:
        for d in rows:
            word = rng.permutation(66)[:w]
            place = rng.permuted(np.tile(np.arange(32), (w, 1)), axis=1)
            per_word = d // w + (np.arange(w) < d % w)
            to = np.concatenate([word[i] * 32 + place[i, :per_word[i]] for i in range(w)])
            assert len(to) == d and len(np.unique(to // 32)) == w
            pairs.append(np.stack([np.full(d, u), to], 1))
            u += 1
    return G.from_edge_pairs(np.concatenate(pairs), n, True)


@pytest.mark.parametrize("words, n", [((31, 32, 33), 3000), ((63, 64, 65), 3000), ((31, 32, 33), 1 << 19),
                                      ((63, 64, 65), (1 << 19) - 1), ((63, 64, 65), 1 << 19)])
def test_words_and_rows_of_owners(device, words, n):
    c = owners_over_hubs(words, (127, 128, 129), n)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    expect = O.triangle_count(c.offsets, c.targets)
    assert g.triangle_count()["total_triangles"] == expect
    b = G.GpuBatch.from_graphs([(c.offsets, c.targets)], device)
    assert b.triangle_count()["total_triangles"].tolist() == [expect]
