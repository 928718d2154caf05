"""GPU test of the deposit's larger tiles: supports so wide that the pairs with 8 x 4
x 4 tiles pass the line of the 8 x 8 x 4 ones, on mesh sides with every kind of
remainder of the tile edges, and, past 2^31 - 1 pairs with those too, the 8^3 tiles
of the CUDA cores."""
import os

import numpy as np
import pytest

from helpers import DEP_TOL

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

L = 64.0


def tiles(nc, x, y, z):
    return -(-nc // x) * -(-nc // y) * -(-nc // z)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nc", [64, 65, 68, 70, 93])
def test_wide_tiles(gpu_ctx, oracle, periodic, nc):
    """Every cell within DEP_TOL of the oracle's FP64 sums of the library's weights
    (v of those of their magnitudes), the FP64 masses within 1e-10."""
    small = 9  # a second mesh of the same deposit
    n = int(1.15 * 8 * 2 ** 20 / tiles(nc, 8, 4, 4))
    if periodic:
        n //= 4  # each reaches most tiles in several images
    rng = np.random.default_rng(nc)
    x = np.minimum(rng.uniform(0, L, (n, 3)), np.nextafter(np.float32(L), np.float32(0))).astype(np.float32)
    # most supports reach all of the mesh, some little
    rk = np.where(rng.uniform(size=n) < 0.9, rng.uniform(1.0, 1.2, n) * L, rng.uniform(0.5, 9.0, n))
    if periodic:
        rk = np.minimum(rk, 0.9 * L)
    rk = rk.astype(np.float32)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    dens = rng.uniform(0.5, 2.0, n).astype(np.float32)
    igrp = rng.choice([-1, 0, 0, 2], n).astype(np.int32)
    p = api.make_particles(x, v, dens=dens, rk=rk, igrp=igrp)
    meshes, tot = gpu_ctx.assign_on_meshes(p, L, [small, nc], -1, periodic=periodic)
    assert gpu_ctx.deposit_stats()["buckets"] == tiles(small, 8, 8, 4) + tiles(nc, 8, 8, 4)
    how = {"periodic": periodic, "offset": (0.0, 0.0, 0.0), "float_weights": True,
           "nthreads": os.cpu_count() or 1}
    for c, got, t in zip((small, nc), meshes, tot):
        nm = c ** 3
        _, s64, t64 = oracle.assign_on_mesh(x, v, dens, rk, igrp, L, c, -1, **how)
        _, a64, _ = oracle.assign_on_mesh(x, np.abs(v), dens, rk, igrp, L, c, -1, **how)
        a64[:3 * nm] = s64[:3 * nm]
        assert np.all(np.abs(got - s64) <= DEP_TOL * np.maximum(a64, np.r_[np.zeros(3 * nm), np.repeat(s64[:nm], 3)]))
        for k in range(2):
            assert abs(t[k] - t64[k]) <= 1e-10 * abs(t64[k])


def test_more_pairs_than_numbers(gpu_ctx):
    """32,769 particles that reach all of a 256^3 mesh: 2^31 + 2^16 pairs with the
    wider tiles.  n against FP64 products of the exact 1-D weights, 1e-5 (the accuracy
    bar of the other deposit tests)."""
    torch = pytest.importorskip("torch")
    n, nc = 32769, 256
    rng = np.random.default_rng(1)
    x = rng.uniform(0, L * 0.999, (n, 3)).astype(np.float32)
    rk = rng.uniform(1.05, 1.5, n).astype(np.float32) * np.float32(L)
    p = api.make_particles(x, rk=rk)
    got, tot = gpu_ctx.assign_on_mesh(p, L, nc, -1)
    assert gpu_ctx.deposit_stats()["buckets"] == tiles(nc, 8, 8, 8)
    edges = torch.arange(nc + 1, dtype=torch.float64, device="cuda") * (L / nc)
    h = torch.as_tensor(rk).cuda().double()[:, None]

    def weights(a):
        t = ((edges - torch.as_tensor(x[:, a].copy()).cuda().double()[:, None]) / h).clamp(-1.0, 1.0)
        return (t - 0.5 * t * t.abs()).diff(dim=1)

    wx, wy, wz = (weights(a) for a in range(3))
    out = torch.as_tensor(got[:nc ** 3]).cuda().double().view(nc, nc * nc)
    total = 0.0
    for z in range(0, nc, 16):
        want = ((wz[:, z:z + 16, None] * wy[:, None, :]).reshape(n, -1).T @ wx).view(-1, nc * nc)
        assert ((out[z:z + 16] - want).abs() <= 1e-5 * want).all()
        total += float(want.sum())
    assert abs(tot[0] - total) <= 1e-6 * total  # sums of float weights, good to a few 1e-7 each
