"""GPU test of the merge with the CUDA-core deposit (ASG_DEPOSIT=simt, read once per
process, hence a child): a tile with many work items, cells shared by several blocks.
Its weights are float products of three, so a cell and a mass are within two roundings
(2^-23) of the oracle's FP64 sums of the library's weights, a cell with those of its own
sum on top (DEP_TOL)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from helpers import DEP_TOL

pytestmark = pytest.mark.gpu

L = 64.0

CHILD = """
import sys
import numpy as np
from asmooth_gb300 import api
a = np.load(sys.argv[1])
nc = int(a["nc"])
with api.Context(0) as ctx:
    ctx.load_particles(api.make_particles(a["x"], a["v"], dens=a["dens"], rk=a["rk"], igrp=a["igrp"]), 0.0, 64.0)
    out = {}
    for alone in (0, 1):
        out["tot%d" % alone] = np.ravel(ctx.run_deposit(64.0, [nc], -1, density_only=bool(alone)))
        out["mesh%d" % alone] = ctx.copy_mesh(0, nc ** 3 * (1 if alone else 6))
np.savez(sys.argv[2], **out)
"""


@pytest.mark.parametrize("n,nc", [(600, 8), (40000, 23)])
def test_simt_tile_of_many_items(oracle, tmp_path, n, nc):
    rng = np.random.default_rng(n + nc)
    x = L * 0.9 + rng.normal(0, 0.4, (n, 3))
    x[:50] = rng.uniform(0, L, (50, 3))
    x = np.clip(x, 0, np.nextafter(np.float32(L), np.float32(0))).astype(np.float32)
    v = rng.normal(size=(n, 3)).astype(np.float32)
    dens, rk = (rng.uniform(0.2, 2.0, n).astype(np.float32) for _ in range(2))
    igrp = rng.choice([-1, 0, 0, 2], n).astype(np.int32)
    np.savez(tmp_path / "in.npz", x=x, v=v, dens=dens, rk=rk, igrp=igrp, nc=nc)
    r = subprocess.run([sys.executable, "-c", CHILD, str(tmp_path / "in.npz"), str(tmp_path / "out.npz")],
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       env={**os.environ, "ASG_DEPOSIT": "simt"}, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    got = np.load(tmp_path / "out.npz")
    _, s64, t64 = oracle.assign_on_mesh(x, v, dens, rk, igrp, L, nc, -1, float_weights=True)
    nm = nc ** 3
    for alone in (0, 1):
        for k in range(1 if alone else 3):
            s = s64[k * nm:(k + 1) * nm]
            assert np.all(np.abs(got["mesh%d" % alone][k * nm:(k + 1) * nm] - s) <= DEP_TOL * np.abs(s)), k
        for k in range(1 if alone else 2):
            assert abs(got["tot%d" % alone][k] - t64[k]) <= 2.0 ** -23 * abs(t64[k])
