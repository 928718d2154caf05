"""GPU test of the deposit's tiles, entries and work items: mesh sides on both
sides of the tile edges (8 x 4 x 4 cells, 8^3 for density alone), bundles of 32
particles that are partial, that share their tiles, that reach many, and that
lie far apart in a mesh they hardly touch, and tiles of one and of many work
items, in the plain, periodic and density-only deposits.  Every cell is within
DEP_TOL of the oracle's FP64 sums of the library's weights, the FP64 masses
within 1e-10."""
import numpy as np
import pytest

from helpers import DEP_TOL

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

L = 64.0


def particles(kind, n, nc):
    rng = np.random.default_rng(1000 * n + nc)
    if kind == "shared":  # all in a few cells: one tile, many work items
        x = 20.0 + rng.normal(0, 1.0, (n, 3))
        rk = rng.uniform(0.2, 1.0, n)
    elif kind == "wide":  # supports over a large part of the mesh
        x = rng.uniform(0, L, (n, 3))
        rk = rng.uniform(2.0, 25.0, n)
    else:  # far: a pair of particles near each of the corners, tiny supports
        x = rng.integers(0, 2, (n, 3)) * (L - 2.0) + rng.uniform(0.5, 1.5, (n, 3))
        rk = rng.uniform(0.01, 0.05, n)
    return (np.clip(x, 0, np.nextafter(np.float32(L), np.float32(0))).astype(np.float32),
            rng.normal(size=(n, 3)).astype(np.float32), rng.uniform(0.5, 2.0, n).astype(np.float32),
            rk.astype(np.float32), rng.choice([-1, 0, 0, 2], n).astype(np.int32))


@pytest.mark.parametrize("mode", ["plain", "periodic", "density"])
@pytest.mark.parametrize("kind,n,nc", [("shared", 1, 8), ("shared", 33, 9), ("shared", 5000, 16),
                                       ("wide", 31, 7), ("wide", 100, 33), ("wide", 1000, 20),
                                       ("far", 64, 33), ("far", 95, 70)])
def test_deposit_tiles(gpu_ctx, oracle, mode, kind, n, nc):
    x, v, dens, rk, igrp = particles(kind, n, nc)
    p = api.make_particles(x, v, dens=dens, rk=rk, igrp=igrp)
    periodic = mode == "periodic"
    _, s64, t64 = oracle.assign_on_mesh(x, v, dens, rk, igrp, L, nc, -1, periodic=periodic,
                                        offset=(0.0, 0.0, 0.0), float_weights=True)
    nm = nc ** 3
    if mode == "density":
        got = gpu_ctx.assign_on_density_mesh(p, L, nc, -1)
        assert np.all(np.abs(got - s64[:nm]) <= DEP_TOL * np.abs(s64[:nm]))
        return
    if periodic:
        got, tot = gpu_ctx.assign_on_global_mesh(p, L, nc, -1)
    else:
        got, tot = gpu_ctx.assign_on_mesh(p, L, nc, -1)
    for k in range(3):
        s = s64[k * nm:(k + 1) * nm]
        assert np.all(np.abs(got[k * nm:(k + 1) * nm] - s) <= DEP_TOL * np.abs(s)), k
    scale = np.abs(s64[3 * nm:]) + np.repeat(s64[:nm], 3)
    # v sums signed terms: the bound holds against the sum of their magnitudes
    _, a64, _ = oracle.assign_on_mesh(x, np.abs(v), dens, rk, igrp, L, nc, -1, periodic=periodic,
                                      offset=(0.0, 0.0, 0.0), float_weights=True)
    scale = np.maximum(scale, a64[3 * nm:])
    assert np.all(np.abs(got[3 * nm:] - s64[3 * nm:]) <= DEP_TOL * scale)
    for k in range(2):
        assert abs(tot[k] - t64[k]) <= 1e-10 * abs(t64[k])
