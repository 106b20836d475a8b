"""Batched PageRank where the mass is not 1: unions that are not symmetric are
pulled over their own lists, which multiplies it, and a damping outside [0, 1]
makes it grow or negative. Iterations, convergence and ranks against the FP64
oracle; and the dangling mass of seeds without entries, repeated ones among them."""
from __future__ import annotations

import math

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def csr(pairs, n, symmetric):
    c = G.from_edge_pairs(np.asarray(pairs), n, symmetric)
    return c.offsets, c.targets


def fan(n):
    """0 and 1 list each other, n more vertices list one of them: each takes its rank, whole."""
    return csr([(0, 1), (1, 0)] + [(v, v % 2) for v in range(2, n + 2)], n + 2, False)


def holed(n, seed):
    """A random symmetric graph whose every third vertex has no entries."""
    p = np.random.default_rng(seed).integers(0, n, size=(4 * n, 2))
    return csr(p[(p % 3 != 0).all(1)], n, True)


def run(device, members, seeds, damping, iterations, tolerance):
    b = G.GpuBatch.from_graphs(members, device)
    b.set_pagerank_seeds(np.asarray(seeds), damping, iterations, tolerance)
    r = b.personalized_pagerank()
    vb = b.vertex_base
    return r, [r["ranks"][vb[g]:vb[g + 1]].astype(np.float64) for g in range(len(members))]


def tele(m, seeds):
    return O.seed_vector(len(m[0]) - 1, seeds)


# A rank is rounded to FP32 twice an iteration (rank and contribution). A vertex of
# the fan follows the 2-cycle, whose errors the damping shrinks by 0.85 a step; its
# own rank adds two more. Relative, as all terms are positive.
FAN_RTOL = 2 * 2.0**-24 / 0.15 + 2 * 2.0**-24


@pytest.mark.parametrize("tolerance", [300.0, 3.0, 0.4, 0.05])
def test_changes_far_above_one(device, tolerance):
    members = [fan(1000), holed(300, 1), fan(37), fan(4000)]
    seeds = [[0], [1], [0], [0]]
    r, ranks = run(device, members, seeds, 0.85, 200, tolerance)
    for g, m in enumerate(members):
        ref = O.pagerank(*m, 0.85, 200, tolerance, tele=tele(m, seeds[g]))
        assert (r["iterations"][g], bool(r["converged"][g])) == (ref["iterations"], ref["converged"]), g
        assert np.allclose(ranks[g], ref["ranks"], rtol=FAN_RTOL, atol=1e-7), g


@pytest.mark.parametrize("damping", [1.5, 2.0, -0.5, -1.5, 1.0, 0.0])
def test_damping_outside_the_unit_interval(device, damping):
    members = [holed(300, 2), holed(64, 3), fan(50)]
    seeds = [[0, 4, 3], [3, 6, 9], [0, 1, 2]]  # multiples of 3: no entries
    r, ranks = run(device, members, seeds, damping, 25, 1e-6)
    for g, m in enumerate(members):
        ref = O.pagerank(*m, damping, 25, 1e-6, tele=tele(m, seeds[g]))
        assert bool(r["converged"][g]) == ref["converged"], g
        if not ref["converged"]:
            assert r["iterations"][g] == ref["iterations"] == 25
        # The terms have both signs: errors relative to the sum of the magnitudes, growing with
        # |damping| > 1 as the ranks themselves do, each iteration adding two roundings.
        mag = np.abs(ref["ranks"]).sum()
        assert np.abs(ranks[g] - ref["ranks"]).sum() <= 4 * 25 * 2.0**-24 * mag + 1e-6, g


def test_no_number_never_converges(device):
    members = [holed(100, 4), fan(10)]
    for damping in (math.nan, math.inf):
        r, _ = run(device, members, [[1], [0]], damping, 7, 1e-6)
        assert r["iterations"].tolist() == [7, 7] and not r["converged"].any()


def test_tolerances_without_a_scale(device):
    members = [holed(100, 5), fan(10), csr(np.zeros((0, 2), np.int64), 4, True)]
    seeds = [[1], [0], [2]]
    for tolerance in (0.0, -1.0, math.nan):
        r, _ = run(device, members, seeds, 0.85, 9, tolerance)
        assert r["iterations"].tolist() == [9, 9, 9] and not r["converged"].any(), tolerance
    r, _ = run(device, members, seeds, 0.85, 9, math.inf)
    assert r["iterations"].tolist() == [1, 1, 1] and r["converged"].all()
    r, _ = run(device, members, seeds, 0.85, 500, 1e-30)  # below any change of an FP32 rank but 0
    assert r["converged"][2]


@pytest.mark.parametrize("per_graph", [1, 2, 5, 33])
def test_seeds_without_entries(device, per_graph):
    rng = np.random.default_rng(per_graph)
    members = [holed(90 + 7 * i, i) for i in range(40)]
    # Multiples of 3 have no entries; repeats and others among them.
    seeds = [[int(3 * rng.integers(0, 5)) + int(rng.integers(0, 9) == 0) for _ in range(per_graph)] for _ in members]
    r, ranks = run(device, members, seeds, 0.85, 60, 1e-6)
    for g, m in enumerate(members):
        n_it = int(r["iterations"][g])
        ref = O.pagerank(*m, 0.85, n_it, 0.0, tele=tele(m, seeds[g]))
        # As in the union passes' tests: two roundings of a total rank of 1 per iteration, damped.
        assert np.abs(ranks[g] - ref["ranks"]).sum() <= 2 * 2.0**-24 / 0.15, g
        want = O.pagerank(*m, 0.85, 60, 1e-6, tele=tele(m, seeds[g]))
        assert abs(n_it - want["iterations"]) <= 1 and bool(r["converged"][g]) == want["converged"], g
