"""GPU test of the search where a bundle's particles lie far apart around a dense
clump, so that its box holds most of the others while each of its radii reaches
few: the 33rd keys equal the oracle's exactly and dens is within 1e-5 of the FP64 sum
over the oracle's lists, with 4, 2 and 1 warps per bundle (in the density 8, 4 and 2),
leaf lists that overflow, and leaves of other sizes."""
import os

import numpy as np
import pytest

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

NTHREADS = os.cpu_count() or 1


@pytest.mark.parametrize("leaf", ["", "5", "32"])
@pytest.mark.parametrize("n,sigma", [(3000, 0.5), (20000, 0.2), (48640, 0.2), (48641, 0.2), (60000, 0.05), (100000, 0.5)])
def test_clump_and_outskirts(oracle, monkeypatch, leaf, n, sigma):
    if leaf:
        monkeypatch.setenv("ASG_LEAF_SIZE", leaf)
    rng = np.random.default_rng(n)
    x = 50.0 + sigma * rng.standard_t(2, (n, 3))  # heavy tails
    x = np.clip(x, 0.0, 99.9).astype(np.float32)
    x[x >= 99.9] = rng.uniform(0, 99.9, (x >= 99.9).sum())
    x[x <= 0.0] = rng.uniform(0, 99.9, (x <= 0.0).sum())
    with api.Context(0) as ctx:
        p = api.make_particles(x)
        ctx.neighbor_search(p, 0.0, 100.0)
        t33, idx33 = ctx.get_knn(n)
    te, ie, nbr = oracle.knn_exact(x, 0.0, 100.0, NTHREADS)
    assert np.array_equal(t33.view(np.int32), te.view(np.int32))
    assert np.array_equal(idx33, ie)
    _, _, d64 = oracle.dens_from_lists(x, nbr, te)
    assert np.max(np.abs(p["dens"] - d64) / d64) <= 1e-5


@pytest.mark.parametrize("n,sigma,ll", [(20000, 0.2, 0.002), (100000, 0.5, 0.004), (100000, 0.5, 0.03)])
def test_groups_of_clump_and_outskirts(gpu_ctx, oracle, n, sigma, ll):
    """FOF with a linking length far below the boxes of the outer bundles, which open
    many nodes: the same groups as the exact oracle."""
    import pyoracle as po

    rng = np.random.default_rng(n)
    x = np.clip(50.0 + sigma * rng.standard_t(2, (n, 3)), 0.0, 99.9).astype(np.float32)
    p = api.make_particles(x)
    ng = gpu_ctx.group_fof(p, 0.0, 100.0, ll)
    lab, want = oracle.group_fof(x, 0.0, 100.0, np.float32(ll), exact=True)
    assert ng == want
    assert np.array_equal(po.canonical_groups(p["igrp"]), po.canonical_groups(lab))


@pytest.mark.parametrize("leaf", ["", "5", "32"])
@pytest.mark.parametrize("n,ll", [(33, 0.5), (40000, 0.02), (150000, 0.1), (150000, 0.4)])
def test_groups_of_a_sheet(oracle, monkeypatch, leaf, n, ll):
    """FOF in a thin sheet across the middle of the box, which the curve leaves and
    enters again, so that some bundles' boxes span a part of it."""
    import pyoracle as po

    if leaf:
        monkeypatch.setenv("ASG_LEAF_SIZE", leaf)
    rng = np.random.default_rng(n)
    x = rng.uniform(0, 100.0, (n, 3))
    x[:, 2] = 50.0 + 0.1 * rng.normal(size=n)
    x = np.clip(x, 0.0, 99.99).astype(np.float32)
    p = api.make_particles(x)
    with api.Context(0) as ctx:
        ng = ctx.group_fof(p, 0.0, 100.0, ll)
    lab, want = oracle.group_fof(x, 0.0, 100.0, np.float32(ll), exact=True)
    assert ng == want
    assert np.array_equal(po.canonical_groups(p["igrp"]), po.canonical_groups(lab))
