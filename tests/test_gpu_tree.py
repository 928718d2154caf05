"""GPU tests of the blocked box tree at the sizes where its shape changes (a
partial last leaf, one and two boxes above 32, a second level) and where the
index sort takes one tile more (multiples of 3072), for leaf sizes on both
sides of 16: 33rd keys and FOF groups equal the oracle's exactly,
dens is within 1e-5 of the FP64 sum over the oracle's lists."""
import os

import numpy as np
import pytest

import pyoracle as po
from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

NTHREADS = os.cpu_count() or 1


def points(n, seed):
    """Half uniform, half in a cluster 1000 times as dense, and one far corner:
    bundles across the cluster's edge reach more leaves than a list holds."""
    rng = np.random.default_rng(seed)
    x = rng.uniform(0, 10, (n, 3))
    x[: n // 2] = 5.0 + rng.normal(0, 0.3, (n // 2, 3))
    return np.clip(x, 0, 9.999).astype(np.float32)


@pytest.mark.parametrize("leaf", ["", "5", "17", "32"])
@pytest.mark.parametrize("n", [33, 47, 511, 513, 1056, 3072, 3073, 16385, 17000])
def test_tree_shapes(oracle, monkeypatch, leaf, n):
    if leaf:
        monkeypatch.setenv("ASG_LEAF_SIZE", leaf)
    x = points(n, 100 + n)
    with api.Context(0) as ctx:
        p = api.make_particles(x)
        ctx.neighbor_search(p, 0.0, 10.0)
        t33, idx33 = ctx.get_knn(n)
        te, ie, nbr = oracle.knn_exact(x, 0.0, 10.0, NTHREADS)
        assert np.array_equal(t33.view(np.int32), te.view(np.int32))
        assert np.array_equal(idx33, ie)
        _, _, d64 = oracle.dens_from_lists(x, nbr, te)
        assert np.max(np.abs(p["dens"] - d64) / d64) <= 1e-5
        q = api.make_particles(x)
        ll = np.float32(0.3)
        ng = ctx.group_fof(q, 0.0, 10.0, ll)
        lab, ng_ref = oracle.group_fof(x, 0.0, 10.0, ll, exact=True)
        assert ng == ng_ref
        assert np.array_equal(po.canonical_groups(q["igrp"]), po.canonical_groups(lab))
