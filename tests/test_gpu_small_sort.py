"""GPU tests of the index at the sizes where its sort changes (one cluster of 8
blocks, of 16 with 1 and 2 elements per thread, many blocks): with the
particles in an order that the sort has to undo and half of them in ties, the
33rd keys equal the oracle's exactly, and the input order does not show in the
result: rk of a shuffled set is the shuffled rk."""
import os

import numpy as np
import pytest

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

NTHREADS = os.cpu_count() or 1
EDGES = [1023, 8191, 8192, 8193, 16384, 16385, 32768, 32769, 65536, 65537]


@pytest.mark.parametrize("n", EDGES)
def test_sort_sizes(oracle, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 10, (n, 3)).astype(np.float32)
    x[n // 2:] = np.round(x[n // 2:] * 4) / 4  # lattice points, many equal keys
    x = np.minimum(x, np.float32(9.999))
    order = rng.permutation(n)
    with api.Context(0) as ctx:
        p = api.make_particles(x)
        ctx.neighbor_search(p, 0.0, 10.0)
        t33, idx33 = ctx.get_knn(n)
        te, ie, _ = oracle.knn_exact(x, 0.0, 10.0, NTHREADS)
        assert np.array_equal(t33.view(np.int32), te.view(np.int32))
        assert np.array_equal(idx33, ie)
        assert (p["rk"] > 0).all()
        q = api.make_particles(x[order])
        ctx.neighbor_search(q, 0.0, 10.0)
    assert np.array_equal(q["rk"], p["rk"][order])
