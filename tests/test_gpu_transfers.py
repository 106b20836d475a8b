"""Large host arrays to the device and back: the staged copies' chunk edges.

Sizes lie around the 1 MB slots and the limits from which copies are staged
(4 MB down, 16 MB up; 64 MB up takes more workers, and fills all slots). Every
value comes back as it went in.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

MB = 1 << 18  # entries


def lists(entries: int, seed: int) -> tuple[np.ndarray, np.ndarray]:
    """A CSR of `entries` sorted entries in lists of up to 61, and its vertex count below 2^26."""
    lengths = np.full(entries // 61 + 2, 61, dtype=np.int64)
    offsets = np.minimum(np.concatenate([[0], np.cumsum(lengths)]), entries).astype(np.uint32)
    row = np.repeat(np.arange(len(lengths), dtype=np.int64), np.diff(offsets))
    n = len(lengths)
    step = max(1, n // 64)
    start = (np.arange(n, dtype=np.int64) * (2 * seed + 1)) % step
    targets = start[row] + (np.arange(entries) - offsets[row]) * step
    keep = targets < n
    counts = np.bincount(row[keep], minlength=n)
    return np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32), targets[keep].astype(np.uint32)


def back(g) -> tuple[np.ndarray, np.ndarray]:
    csr = g.to_csr()
    return csr.offsets, csr.targets


@pytest.mark.parametrize("entries", [MB - 1, MB + 1, 4 * MB, 4 * MB + 1, 16 * MB - 1, 16 * MB + 3, 64 * MB - 5,
                                     65 * MB + 1, 150 * MB + 7])
def test_csr_round_trip(device, entries):
    o, t = lists(entries, entries % 11)
    ro, rt = back(G.GpuGraph.from_csr(o, t, device))
    assert np.array_equal(ro, o) and np.array_equal(rt, t)


def test_threads_share_the_slots(device):
    """Uploads and downloads of one device from several threads at once."""
    cases = [lists(20 * MB + 17 * i, i) for i in range(4)]
    bad = []

    def work(i):
        o, t = cases[i]
        for _ in range(3):
            ro, rt = back(G.GpuGraph.from_csr(o, t, device))
            if not (np.array_equal(ro, o) and np.array_equal(rt, t)):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not bad


def test_pairs_and_edge_list(device):
    """From pairs above the upload limit; a kept edge list outlives its graph and other lists."""
    rng = np.random.default_rng(5)
    pairs = rng.integers(0, 4000, size=(2_300_001, 2), dtype=np.uint32)
    g = G.GpuGraph.from_edge_pairs(pairs, 4000, True, device)
    o, t = O.from_edge_pairs(pairs, 4000, True)[:2]
    ro, rt = back(g)
    assert np.array_equal(ro, o) and np.array_equal(rt, t)
    first = g.k_truss_array(3)["edges"]
    tail = first[-5:]
    expected = O.k_truss(o, t, 3)["edges"]
    second = g.k_truss_array(3)["edges"]
    second[:] = 0  # a list of its own
    del g, second
    assert first.dtype == np.uint32 and first.flags.c_contiguous and first.flags.writeable
    assert np.array_equal(first, expected)
    del first
    assert np.array_equal(tail, expected[-5:])
    assert G.GpuGraph.from_edge_pairs(pairs[:2], 4000, True, device).k_truss_array(3)["edges"].shape == (0, 2)
