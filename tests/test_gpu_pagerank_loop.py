"""PageRank's one-launch loop at the shapes where its phases meet: no long rows,
only a few, chunks of 256 one-entry rows, rows that cross many chunks, rows of
exactly 1,024 entries, dangling vertices, runs of 0 and 1 iterations and runs of
more than one launch (512 iterations)."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# Ranks and contributions are FP32, sums FP64 (long rows: compensated FP32): a
# rounding of at most 2^-24 of a total rank of 1 in each, damped by 0.85 a step.
L1 = 2 * 2.0**-24 / 0.15


def graph(name):
    rng = np.random.default_rng(7)
    if name == "pairs":  # one-entry rows only
        n = 3001
        return np.stack([np.arange(0, n - 1, 2), np.arange(1, n, 2)], 1), n
    if name.startswith("star"):
        n = int(name[4:])
        return np.stack([np.zeros(n, np.int64), np.arange(1, n + 1)], 1), n + 3
    if name == "rows":  # long rows and rows that cross chunks, side by side
        out, at = [], 0
        for k in (255, 256, 257, 600, 1023, 1024, 1025, 2048, 5000):
            out.append(np.stack([np.full(k, at), np.arange(at + 1, at + 1 + k)], 1))
            at += k + 1
        return np.concatenate(out), at
    n, m = (int(x) for x in name.split("x"))
    return rng.integers(0, n, size=(m, 2)), n


@pytest.mark.parametrize("name", ["pairs", "star1023", "star1024", "star70000", "rows", "5x9", "1000x300",
                                  "3000x200000", "100003x400000"])
@pytest.mark.parametrize("directed", [False, True])
def test_loop_matches_oracle(device, name, directed):
    pairs, n = graph(name)
    c = G.from_edge_pairs(pairs, n, not directed)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    for iterations in (0, 1, 23):
        if directed:
            r = g.pagerank_directed(0.85, iterations, 0.0)
            ref = O.pagerank_directed(c.offsets, c.targets, 0.85, iterations, 0.0)
        else:
            r = g.pagerank_array(0.85, iterations, 0.0)
            ref = O.pagerank(c.offsets, c.targets, 0.85, iterations, 0.0)
        assert r["iterations"] == iterations and not r["converged"]
        assert np.abs(r["ranks"].astype(np.float64) - ref["ranks"]).sum() <= L1, iterations


def test_runs_of_several_launches(device):
    pairs, n = graph("1000x300")
    c = G.from_edge_pairs(pairs, n, True)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    ref = O.pagerank(c.offsets, c.targets, 0.85, 1100, 0.0)
    for _ in range(2):
        r = g.pagerank_array(0.85, 1100, 0.0)
        assert r["iterations"] == 1100 and not r["converged"]
        assert np.abs(r["ranks"].astype(np.float64) - ref["ranks"]).sum() <= L1
    for damping, tolerance in ((0.999, 1e-4), (0.85, 1e-4)):  # ends as the oracle's run ends
        r = g.pagerank_array(damping, 1100, tolerance)
        ref = O.pagerank(c.offsets, c.targets, float(np.float32(damping)), 1100, tolerance)
        assert (r["converged"], r["iterations"]) == (ref["converged"], ref["iterations"])
