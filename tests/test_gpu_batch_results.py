"""Results of a batch on which only some of the calls have run: those that have
not run are not asked for, and do not fail."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import grafeo_cuda as G
from grafeo_cuda._lib import check, lib

pytestmark = pytest.mark.gpu

K4 = (np.array([0, 3, 6, 9, 12], np.uint32), np.array([1, 2, 3, 0, 2, 3, 0, 1, 3, 0, 1, 2], np.uint32))


def triangles(b):
    tri = np.zeros(b.num_graphs, dtype=np.uint64)
    check(lib.gcu_batch_results(b._h, tri.ctypes.data_as(C.POINTER(C.c_uint64)), None, None, None, None, None, None))
    return tri


def test_triangles_alone(device):
    # The pool hands the batch the memory of small freed graphs, whose words are not zero.
    for turn in range(20):
        graphs = [G.GpuGraph.from_csr(*K4, device) for _ in range(64)]
        for g in graphs:
            g.bfs_array(0)
        del graphs, g
        b = G.GpuBatch.from_graphs([K4, K4], device)
        assert b.triangle_count()["total_triangles"].tolist() == [4, 4]
        assert triangles(b).tolist() == [4, 4], turn
        b.set_bfs_sources(np.zeros((2, 1), np.uint32))
        assert triangles(b).tolist() == [4, 4], turn
        b.bfs()
        b.set_pagerank_seeds(np.zeros((2, 1), np.uint32))
        assert triangles(b).tolist() == [4, 4], turn
