"""GPU test that after asg_neighbor_search_noalloc's preparing call no particle count
takes device memory: the sort, the search and the density run other kernels for other
counts.  In a process of its own, where nothing has loaded them before."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes as C
import torch
from asmooth_gb300 import _lib
lib = _lib.load()
N = 32768
x = torch.rand((N, 3), device="cuda")
rk, dens = torch.zeros(N, device="cuda"), torch.zeros(N, device="cuda")
torch.cuda.synchronize()
assert lib.asg_neighbor_search_noalloc(None, 0, 0.0, 0.0, None, None, None) == 0
p = [C.c_void_p(t.data_ptr()) for t in (x, rk, dens)]
free = torch.cuda.mem_get_info()[0]
for n in (33, 8192, 8193, 16384, 16385, 24320, 24321, 32768):
    assert lib.asg_neighbor_search_noalloc(p[0], n, 0.0, 1.0, p[1], p[2], None) == 0, n
    assert torch.cuda.mem_get_info()[0] == free, n
"""


def test_no_particle_count_takes_memory_after_the_preparing_call():
    pytest.importorskip("torch")
    from asmooth_gb300 import build as B

    B.build()
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
