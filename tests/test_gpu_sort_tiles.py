"""Device CSR builds where a block of the radix sort takes more than one tile of
2,048 keys: up to seven waves of four blocks per SM take one tile each, beyond them
every block takes two, the last one fewer where the tiles do not go up. The CSR
equals numpy's sort of the pairs."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import grafeo_cuda as G

pytestmark = pytest.mark.gpu

TILE = 2048


def numpy_csr(p, n):
    keys = np.unique(p[:, 0].astype(np.uint64) << np.uint64(32) | p[:, 1].astype(np.uint64))
    offsets = np.zeros(n + 1, dtype=np.uint64)
    np.cumsum(np.bincount((keys >> np.uint64(32)).astype(np.int64), minlength=n), out=offsets[1:])
    return offsets.astype(np.uint32), (keys & np.uint64(0xFFFFFFFF)).astype(np.uint32)


@pytest.mark.parametrize("extra", [-1, 0, 1, TILE, TILE + 1, 2 * TILE - 1, 2 * TILE + 5])
def test_tiles_per_block(device, extra):
    one_each = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 7
    m, n = one_each * TILE + extra, 300_007
    p = np.random.default_rng(extra + 1).integers(0, n, size=(m, 2), dtype=np.uint32)
    csr = G.GpuGraph.from_edge_pairs(p, n, False, device).to_csr()
    o, t = numpy_csr(p, n)
    assert np.array_equal(csr.offsets, o) and np.array_equal(csr.targets, t)
