"""GPU check of the radix sort's 64-bit tile states, which only 2^30 and more elements
take: tests/gpu_checks/sort_check.cu is compiled for sm_103a here and run once."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


def test_sort_with_wide_states(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "sort_check"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-o", str(exe),
                    os.path.join(HERE, "gpu_checks", "sort_check.cu")], check=True, capture_output=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    lines = r.stdout.strip().splitlines()
    assert len(lines) == 21, r.stdout + r.stderr
    assert all("mismatches 0 error word 0 no error" in ln for ln in lines), r.stdout
    assert r.returncode == 0
