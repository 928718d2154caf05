"""GPU test of a context after its batch was tuned: the set that the tuner leaves
loaded (the largest item) answers as if it had been loaded by itself, from whatever
leaf size the context started, and a later, larger batch of the same context gives
what asg_smooth gives."""
import numpy as np
import pytest

from asmooth_gb300 import api
from asmooth_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def bits(a):
    return np.asarray(a, np.float32).view(np.int32)


@pytest.mark.parametrize("leaf", ["", "32"])
def test_context_after_tuning(monkeypatch, leaf):
    if leaf:
        monkeypatch.setenv("ASG_LEAF_SIZE", leaf)
    items, ncs = syn.make_batch(scale=4, n_cubes=2)
    items = sorted(items, key=lambda c: c.n)
    with api.Context(0) as ctx, api.Context(0) as ref:
        for cubes in (items[:1], items[-2:]):
            with api.Batch(ctx, cubes, ncs) as b:
                b.tune()
                big = cubes[-1]
                ref.load_particles(api.make_particles(big.x, big.v), big.left, big.right)
                ref.run_neighbor_search()
                for ours, theirs in zip(ctx.get_knn(big.n), ref.get_knn(big.n)):
                    assert np.array_equal(ours, theirs)
                halos = api.make_halos([[big.boxsize / 2] * 3], [big.boxsize / 4], [1.0])
                assert ctx.run_mark_halos(halos) == ref.run_mark_halos(halos)
                assert ctx.run_fof(0.8) == ref.run_fof(0.8)
                b.run()
                for i, cube in enumerate(cubes):
                    rk, dens, _, _ = b.get(i)
                    p = api.make_particles(cube.x, cube.v)
                    ref.smooth(p, cube.left, cube.right, cube.boxsize, ncs, -1)
                    assert np.array_equal(bits(rk), bits(p["rk"]))
                    assert np.max(np.abs(dens - p["dens"]) / p["dens"]) <= 1e-5
