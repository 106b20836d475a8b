"""k-trusses of graphs of one device from several threads at once. The supports'
blocks hold a bitmap as large as the graph has vertices, so the threads launch
one kernel with different amounts of shared memory. Edges and rounds are whole
numbers: equal to the oracle's."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_graphs_of_different_sizes_from_several_threads(device):
    # 76, 119, 154 and 207 KB of bitmap: the 1024-thread form.
    cases = []
    for i, n in enumerate((610_000, 950_000, 1_230_000, 1_650_000)):
        rng = np.random.default_rng(i)
        pairs = rng.integers(0, 3000, size=(40_000, 2)) * (n // 3000)
        c = G.from_edge_pairs(pairs, n, True)
        cases.append((c.offsets, c.targets, O.k_truss(c.offsets, c.targets, 4)))
    bad = []

    def work(i):
        o, t, ref = cases[i]
        try:
            for _ in range(60):  # the supports are a graph's own: a new one each time
                r = G.GpuGraph.from_csr(o, t, device).k_truss_array(4)
                if not np.array_equal(r["edges"], ref["edges"]) or r["iterations"] != ref["iterations"]:
                    bad.append((i, "differs"))
        except Exception as e:  # noqa: BLE001
            bad.append((i, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not bad, bad[:3]
