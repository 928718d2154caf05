"""GPU test of the FOF catalogue at the sizes where its kernels change: halos of
0 to 1025 members (a warp's and a block's chunks, with remainders, and the step
from one to the other at 512) and label sorts of one tile of 4096 and one more,
with 8- and 9-bit digits.  The float sums follow the caller's array order, so
the records equal the oracle's bit for bit only if the sort is stable."""
import numpy as np
import pytest

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

SIZES = [1, 0, 31, 32, 33, 255, 256, 257, 511, 512, 513, 768, 1025, 0]


@pytest.mark.parametrize("extra", [0, 300])  # further halos of one member: 9-bit digits
@pytest.mark.parametrize("n", [sum(SIZES) + 300, 8191, 8192, 8193, 12289])
def test_catalogue_sizes(gpu_ctx, oracle, n, extra):
    rng = np.random.default_rng(n + extra)
    labels = np.repeat(np.arange(1, len(SIZES) + 1), SIZES)
    labels = np.concatenate([labels, len(SIZES) + 1 + np.arange(extra)])
    igrp = np.zeros(n, np.int32)
    igrp[:len(labels)] = labels
    igrp = igrp[rng.permutation(n)]
    p = api.make_particles(rng.uniform(0, 100, (n, 3)), rng.normal(size=(n, 3)), igrp=igrp)
    nhalo = len(SIZES) + extra
    want = oracle.fof_halos(p["x"], p["v"], igrp, nhalo, 100.0)
    assert len(want) == sum(s > 0 for s in SIZES) + extra
    assert gpu_ctx.fof_halos(p, nhalo, 100.0).tobytes() == want.tobytes()
