"""GPU tests of the halo marking where the warps per halo change (4864 halos) and
for leaf sizes that fill half a warp, part of one and all of it: marks, counts
and masses equal a float32 evaluation over all particles exactly."""
import numpy as np
import pytest

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", ["", "5", "24", "32"])
@pytest.mark.parametrize("n,nh", [(40, 1), (1500, 33), (3000, 4864), (3000, 4865)])
def test_marks_equal_direct_test(monkeypatch, leaf, n, nh):
    if leaf:
        monkeypatch.setenv("ASG_LEAF_SIZE", leaf)
    rng = np.random.default_rng(n + nh)
    x = rng.uniform(0, 10, (n, 3)).astype(np.float32)
    c = rng.uniform(-0.5, 10.5, (nh, 3)).astype(np.float32)  # some centres outside
    r = (0.05 * rng.pareto(1.5, nh) + 0.01).clip(max=9).astype(np.float32)
    mass = rng.uniform(1, 9, nh).astype(np.float32)
    inside = ((c > 0) & (c < 10)).all(axis=1)
    want, count = np.zeros(n, bool), np.zeros(nh, np.int64)
    for h in np.flatnonzero(inside):
        d = c[h] - x
        hit = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2] < r[h] * r[h]
        want |= hit
        count[h] = hit.sum()
    with api.Context(0) as ctx:
        ctx.load_particles(api.make_particles(x), 0.0, 10.0)
        ctx.run_neighbor_search()
        halos = api.make_halos(c, r, mass)
        np_halo, m_halo = ctx.run_mark_halos(halos)
        p = ctx.store_particles(api.make_particles(x))
    assert np.array_equal(p["igrp"] == -1, want)
    assert np_halo == count.sum()
    expect = np.float64(0)
    for h in np.flatnonzero(inside):
        expect += np.float64(np.float32(mass[h] / np.float32(8)))
    assert m_halo == pytest.approx(expect, rel=1e-12)
