"""GPU test of the fields' way back to input order on both sides of every line where
its form changes: streaming loads above 40 MB of fields, one field at a time above 80
MB, 2 to 5 slices of a field, and one again above that.  What was loaded comes back
at its own place, every place is written, and nothing beside the fields is."""
import numpy as np
import pytest

from asmooth_gb300 import api

pytestmark = pytest.mark.gpu

MB40, MB80 = 10 << 20, 20 << 20  # particles whose one field fills 40 and 80 MB


@pytest.mark.parametrize("n,fields", [(1000, "rdg"), (MB40, "d"), (MB40 + 1, "g"), (MB40 // 2, "rd"),
                                      (MB40 // 2 + 1, "dg"), (MB80, "d"), (MB80 + 1, "d"), (MB80 // 3 + 1, "rdg"),
                                      (2 * MB80 + 7, "rg"), (5 * MB80, "d"), (5 * MB80 + 1, "g")])
def test_fields_come_back(n, fields):
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.rand((n, 3), device="cuda", generator=g)
    dens = torch.rand(n, device="cuda", generator=g)
    igrp = torch.randint(-5, 1 << 30, (n,), dtype=torch.int32, device="cuda", generator=g)
    out = {k: torch.full((n + 8,), -1, dtype=t, device="cuda") for k, t in
           (("r", torch.float32), ("d", torch.float32), ("g", torch.int32))}
    torch.cuda.synchronize()
    with api.Context(0) as ctx:
        ctx.load_particles_device(x.data_ptr(), n, 0.0, 1.0, dens_ptr=dens.data_ptr(), igrp_ptr=igrp.data_ptr())
        ctx.store_fields_device(*[out[k].data_ptr() if k in fields else 0 for k in "rdg"])
    want = {"r": torch.zeros_like(dens), "d": dens, "g": igrp}
    for k in "rdg":
        if k in fields:
            assert torch.equal(out[k][:n], want[k]) and bool((out[k][n:] == -1).all())
        else:
            assert bool((out[k] == -1).all())
