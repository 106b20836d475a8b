"""A graph holds the buffers of the form of BFS that has run on it, and no others:
per vertex the one-launch search's two item queues (8 bytes each), or two vertex
queues and a degree scan (4 each); the distances and the list of vertices with
edges (4 each) with either."""
from __future__ import annotations

import numpy as np
import pytest

import grafeo_cuda as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

N = 1 << 23


def used() -> int:
    rt = pytest.importorskip("cuda.bindings.runtime")
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert err == rt.cudaError_t.cudaSuccess
    err, value = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    assert err == rt.cudaError_t.cudaSuccess
    return int(value)


@pytest.mark.parametrize("loop, per_vertex", [(True, 24), (False, 20)], ids=["search", "levels"])
def test_buffers_of_one_form(device, loop, per_vertex):
    # A perfect matching of the first half: most vertices have no edge (the list form of the pull).
    a = np.arange(0, N // 2, 2)
    c = G.from_edge_pairs(np.stack([a, a + 1], 1), N, True)
    g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
    device.set_bfs_device_loop(loop)
    try:
        before = used()
        r = g.bfs_array(4)
        held = used() - before
    finally:
        device.set_bfs_device_loop(True)
    assert (r["reachable"], r["max_depth"]) == (2, 1)
    # Bitmaps (four at most), 2 MB of segments, and the pool's rounding.
    assert held <= per_vertex * N + 4 * N // 8 + (3 << 20), held / N


def test_both_forms_in_turn(device):
    c = G.generate_rmat(12, 8, 0.57, 0.19, 0.19, seed=5)
    for order in ([True, False, True], [False, True, False]):
        g = G.GpuGraph.from_csr(c.offsets, c.targets, device)
        try:
            for loop in order:
                device.set_bfs_device_loop(loop)
                for s in (0, 77):
                    r, ref = g.bfs_array(s), O.bfs(c.offsets, c.targets, s)
                    assert np.array_equal(r["distances"], ref["distances"])
        finally:
            device.set_bfs_device_loop(True)
