"""GPU tests of the tie resolution where its form changes (up to 8 tied queries in
a bundle of 32 one at a time, more together): particles on grids from fine
to coarse, so that few to most queries tie at the 33rd distance; the wrong one of
two tied neighbours would change dens by about a per cent: dens is within 1e-5 of
the FP64 sum over the oracle's lists."""
import os

import numpy as np
import pytest

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

NTHREADS = os.cpu_count() or 1


@pytest.mark.parametrize("leaf", ["", "5", "24"])
@pytest.mark.parametrize("grid", [4000, 400, 150, 40])
def test_dens_with_ties(oracle, monkeypatch, leaf, grid):
    if leaf:
        monkeypatch.setenv("ASG_LEAF_SIZE", leaf)
    n = 6000
    rng = np.random.default_rng(grid)
    x = (rng.integers(0, grid, (n, 3)) * (9.99 / grid)).astype(np.float32)
    with api.Context(0) as ctx:
        p = api.make_particles(x)
        ctx.neighbor_search(p, 0.0, 10.0)
    te, _, nbr = oracle.knn_exact(x, 0.0, 10.0, NTHREADS)
    _, _, d64 = oracle.dens_from_lists(x, nbr, te)
    assert np.max(np.abs(p["dens"] - d64) / d64) <= 1e-5
