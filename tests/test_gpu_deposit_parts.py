"""GPU test of the making of the deposit's entries: bundle counts on both sides of
every change in the number of warps that share a bundle (32 up to 1024 particles, then
powers of two from 16 down to 1), with particles spread over the box, in clumps, and at the
seams of the periodic mesh, so that a bundle's particles reach tiles in one row of
more than 32, in few and in many images.  Every cell is within DEP_TOL of the
oracle's FP64 sums of the library's weights (below float32's normal range, of its
smallest normal number), the FP64 masses within 1e-10."""
import os

import numpy as np
import pytest

from helpers import DEP_TOL

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

L = 64.0
TINY = float(np.finfo(np.float32).tiny)


def particles(kind, n, nc):
    rng = np.random.default_rng(7 * n + nc)
    if kind == "spread":
        x = rng.uniform(0, L, (n, 3))
    elif kind == "clumps":
        x = rng.uniform(0, L, (5, 3))[rng.integers(0, 5, n)] + rng.normal(0, 1.5, (n, 3))
    else:  # seams: near the faces, edges and corners of the box
        x = rng.uniform(0, L, (n, 3))
        near = rng.integers(0, 3, (n, 3))
        x = np.where(near == 0, x, np.where(near == 1, 0.02 * x, L - 0.02 * x))
    x = np.clip(x, 0, np.nextafter(np.float32(L), np.float32(0))).astype(np.float32)
    cells = min(600.0, 4e7 / n) ** (1 / 3)  # of a support on average, as the oracle's time allows
    h = rng.uniform(0.3, 0.7, n) * cells * L / nc
    if n < 100:
        h[::7] = 0.6 * L  # and some over more than half of the mesh
    return (x, rng.normal(size=(n, 3)).astype(np.float32), rng.uniform(0.5, 2.0, n).astype(np.float32),
            h.astype(np.float32), rng.choice([-1, 0, 0, 2], n).astype(np.int32))


@pytest.mark.parametrize("mode", ["plain", "periodic", "density"])
@pytest.mark.parametrize("kind,n,nc", [("spread", 6, 280), ("seams", 64, 61), ("seams", 1000, 33), ("seams", 1024, 80), ("seams", 1025, 64),
                                       ("clumps", 8192, 40), ("seams", 8193, 40), ("spread", 16384, 50),
                                       ("seams", 16385, 50), ("spread", 32768, 40), ("seams", 32769, 41),
                                       ("clumps", 65536, 33), ("seams", 65537, 33), ("seams", 131072, 40), ("clumps", 131073, 40),
                                       ("seams", 262145, 33)])
def test_deposit_parts(gpu_ctx, oracle, mode, kind, n, nc):
    x, v, dens, rk, igrp = particles(kind, n, nc)
    p = api.make_particles(x, v, dens=dens, rk=rk, igrp=igrp)
    periodic = mode == "periodic"
    how = {"periodic": periodic, "offset": (0.0, 0.0, 0.0), "float_weights": True,
           "nthreads": os.cpu_count() or 1}
    _, s64, t64 = oracle.assign_on_mesh(x, v, dens, rk, igrp, L, nc, -1, **how)
    nm = nc ** 3
    if mode == "density":
        got = gpu_ctx.assign_on_density_mesh(p, L, nc, -1)
        assert np.all(np.abs(got - s64[:nm]) <= DEP_TOL * np.maximum(np.abs(s64[:nm]), TINY))
        return
    got, tot = (gpu_ctx.assign_on_global_mesh if periodic else gpu_ctx.assign_on_mesh)(p, L, nc, -1)
    for k in range(3):
        s = s64[k * nm:(k + 1) * nm]
        assert np.all(np.abs(got[k * nm:(k + 1) * nm] - s) <= DEP_TOL * np.maximum(np.abs(s), TINY)), k
    # v sums signed terms: the bound holds against the sum of their magnitudes
    _, a64, _ = oracle.assign_on_mesh(x, np.abs(v), dens, rk, igrp, L, nc, -1, **how)
    scale = np.maximum(np.maximum(a64[3 * nm:], np.repeat(s64[:nm], 3)), TINY)
    assert np.all(np.abs(got[3 * nm:] - s64[3 * nm:]) <= DEP_TOL * scale)
    for k in range(2):
        assert abs(tot[k] - t64[k]) <= 1e-10 * abs(t64[k])
