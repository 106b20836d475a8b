"""Graphs uploaded to one device from several threads at once: each upload's
checks wait for its own copy. What is valid is taken and comes back as it went
in, and what is not is refused with its own message, whatever the others do."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import grafeo_cuda as G

pytestmark = pytest.mark.gpu


def test_each_upload_waits_for_its_own_copy(device):
    cases = []
    for i in range(6):
        n = (40, 3000, 20_000, 90_000, 250_000, 700_000)[i]
        c = G.from_edge_pairs(np.random.default_rng(i).integers(0, n, size=(7 * n, 2)), n, True)
        bad = c.targets.copy()
        row = int(np.flatnonzero(np.diff(c.offsets))[-1])
        bad[c.offsets[row + 1] - 1] = n  # the last list ends past the vertices
        cases.append((c.offsets, c.targets, bad, row))
    wrong = []

    def work(i):
        o, t, b, row = cases[i]
        try:
            for turn in range(max(10, 600_000 // len(t))):
                csr = G.GpuGraph.from_csr(o, t, device).to_csr()
                if not (np.array_equal(csr.offsets, o) and np.array_equal(csr.targets, t)):
                    wrong.append((i, turn, "came back different"))
                try:
                    G.GpuGraph.from_csr(o, b, device)
                    wrong.append((i, turn, "taken"))
                except Exception as e:  # noqa: BLE001
                    if f"node {row} " not in str(e):
                        wrong.append((i, turn, str(e)))
        except Exception as e:  # noqa: BLE001
            wrong.append((i, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(cases))]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not wrong, wrong[:3]
