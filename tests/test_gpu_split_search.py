"""GPU tests of the neighbour search and the density at the sizes where the warps
per bundle change (152, 760, 2736 and 4864 bundles of 32), with half of the
particles on lattice points (equal distances at the 33rd) and a dense cluster:
33rd keys equal the oracle's exactly, dens is within 1e-5 of the FP64 sum over
the oracle's lists."""
import os

import numpy as np
import pytest

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

NTHREADS = os.cpu_count() or 1


def points(n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 10, (n, 3))
    step = 10.0 / np.ceil((4 * n) ** (1 / 3))
    x[: n // 2] = np.floor(x[: n // 2] / step) * step + step / 2
    x[n // 2: n // 2 + n // 8] = 3.0 + rng.normal(0, 0.2, (n // 8, 3))
    return np.clip(x, 0, 9.999).astype(np.float32)


@pytest.mark.parametrize("n", [33, 100, 4864, 4865, 24320, 24321, 87552, 87553, 155648, 155649])
def test_warps_per_bundle(oracle, n):
    x = points(n)
    with api.Context(0) as ctx:
        p = api.make_particles(x)
        ctx.neighbor_search(p, 0.0, 10.0)
        t33, idx33 = ctx.get_knn(n)
    te, ie, nbr = oracle.knn_exact(x, 0.0, 10.0, NTHREADS)
    assert np.array_equal(t33.view(np.int32), te.view(np.int32))
    assert np.array_equal(idx33, ie)
    _, _, d64 = oracle.dens_from_lists(x, nbr, te)
    assert np.max(np.abs(p["dens"] - d64) / d64) <= 1e-5
