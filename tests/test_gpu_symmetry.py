"""The symmetry test of a CSR (it decides which algorithms' forms may run) on
graphs that miss one entry, on either side of a pair, or whose surpluses cancel:
truss_decomposition refuses exactly the CSRs that are not symmetric."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from grafeo_cuda import GrafeoCudaError

pytestmark = pytest.mark.gpu


def csr_of(entries, n):
    e = np.unique(np.asarray(entries, dtype=np.int64), axis=0)
    offsets = np.searchsorted(e[:, 0], np.arange(n + 1)).astype(np.uint32)
    return offsets, e[:, 1].astype(np.uint32)


def symmetric(device, entries, n):
    g = G.GpuGraph.from_csr(*csr_of(entries, n), device)
    try:
        g.truss_decomposition()
        return True
    except GrafeoCudaError as e:
        assert "symmetric" in str(e)
        return False


@pytest.mark.parametrize("case", ["whole", "loops", "hub_side", "leaf_side", "equal_degrees", "cancel", "directed_pair"])
def test_symmetry_decides_the_form(device, case):
    n = 900
    rng = np.random.default_rng(3)
    p = rng.integers(1, n, size=(4000, 2))
    star = np.stack([np.zeros(700, np.int64), np.arange(1, 701)], 1)  # vertex 0 is a hub
    p = np.concatenate([p[p[:, 0] != p[:, 1]], star])
    e = np.unique(np.concatenate([p, p[:, ::-1]]), axis=0)
    if case == "whole":
        assert symmetric(device, e, n)
        return
    if case == "loops":
        assert symmetric(device, np.concatenate([e, [[0, 0], [5, 5]]]), n)
        return

    def without(entries, u, v):
        return entries[~((entries[:, 0] == u) & (entries[:, 1] == v))]

    if case == "hub_side":  # 0 -> 7 gone, 7 -> 0 there
        bad = without(e, 0, 7)
    elif case == "leaf_side":
        bad = without(e, 7, 0)
    elif case == "equal_degrees":
        ring = np.stack([np.arange(n), (np.arange(n) + 1) % n], 1)
        bad = without(np.concatenate([ring, ring[:, ::-1]]), 10, 11)
    elif case == "cancel":  # one entry missing from a long list, one from a short one
        bad = without(without(e, 0, 7), 9, 0)
    else:  # two one-way entries between vertices without another edge
        n = 904
        bad = np.concatenate([e, [[900, 901], [903, 902]]])
    assert not symmetric(device, bad, n)
