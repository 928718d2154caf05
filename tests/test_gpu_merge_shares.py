"""GPU test of the merge of a tile with many work items, whose cells several blocks
share: nearly all particles in one tile of each tile shape (8 x 4 x 4 and 8 x 8 x 8
cells), with few particles elsewhere, on meshes that end inside the tile.  Every cell is
within DEP_TOL of the oracle's FP64 sums of the library's weights, the FP64 masses
within 1e-10."""
import numpy as np
import pytest

from helpers import DEP_TOL

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

L = 64.0


@pytest.mark.parametrize("density_only", [False, True])
@pytest.mark.parametrize("n,nc", [(600, 8), (5000, 13), (40000, 16), (40000, 23)])
def test_one_tile_of_many_items(gpu_ctx, oracle, density_only, n, nc):
    rng = np.random.default_rng(n + nc)
    x = L * 0.9 + rng.normal(0, 0.4, (n, 3))
    x[:50] = rng.uniform(0, L, (50, 3))
    x = np.clip(x, 0, np.nextafter(np.float32(L), np.float32(0))).astype(np.float32)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    dens, rk = (rng.uniform(0.2, 2.0, n).astype(np.float32) for _ in range(2))
    igrp = rng.choice([-1, 0, 0, 2], n).astype(np.int32)
    p = api.make_particles(x, v, dens=dens, rk=rk, igrp=igrp)
    gpu_ctx.load_particles(p, 0.0, L)
    tot = np.ravel(gpu_ctx.run_deposit(L, [nc], -1, density_only=density_only))
    got = gpu_ctx.copy_mesh(0, nc ** 3 * (1 if density_only else 6))
    _, s64, t64 = oracle.assign_on_mesh(x, v, dens, rk, igrp, L, nc, -1, float_weights=True)
    nm = nc ** 3
    for k in range(1 if density_only else 3):
        s = s64[k * nm:(k + 1) * nm]
        assert np.all(np.abs(got[k * nm:(k + 1) * nm] - s) <= DEP_TOL * np.abs(s)), k
    for k in range(1 if density_only else 2):
        assert abs(tot[k] - t64[k]) <= 1e-10 * abs(t64[k])
