"""Runs a kernel's own source text on the CPU, one thread after another: for checks
of index arithmetic on inputs that would reach out of range on the device if the
check failed.  Only kernels without barriers or warp operations."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "asmooth_gb300", "csrc")

SHIM = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <climits>
#include <vector>
struct Dim { unsigned x, y, z; };
static Dim threadIdx, blockIdx, blockDim, gridDim;
struct uint2 { unsigned x, y; };
static uint2 make_uint2(unsigned x, unsigned y) { return {x, y}; }
static int __popc(unsigned v) { return __builtin_popcount(v); }
template <class T> static T atomicAdd(T* p, T v) { T o = *p; *p += v; return o; }
static int atomicOr(int* p, int v) { int o = *p; *p |= v; return o; }
using std::max; using std::min;
static void grid_begin() {}
#define __global__ static
#define __launch_bounds__(...)
template <class F> static void run(unsigned blocks, unsigned threads, F kernel)
{
    gridDim = {blocks, 1, 1};
    blockDim = {threads, 1, 1};
    for (unsigned b = 0; b < blocks; ++b)
        for (unsigned t = 0; t < threads; ++t) {
            blockIdx = {b, 0, 0};
            threadIdx = {t, 0, 0};
            kernel();
        }
}
"""


def constants(*names):
    """the named `constexpr int` definitions of the sources"""
    text = "".join(open(os.path.join(CSRC, f)).read() for f in sorted(os.listdir(CSRC))
                   if f.endswith((".cu", ".cuh", ".h")))
    return "".join(re.search(rf"constexpr int {n} = [^;]*;", text).group(0) + "\n" for n in names)


def kernel_text(unit, name):
    text = open(os.path.join(CSRC, unit + ".cu")).read()
    m = re.search(rf"__global__ void [^;{{]*\b{name}\(.*?\n}}\n", text, re.S)
    assert m, name
    return m.group(0)


def run(tmp_path, code):
    """compiles and runs `code` after the shim; its standard output"""
    src, exe = tmp_path / "kernel.cpp", tmp_path / "kernel"
    src.write_text(SHIM + code)
    subprocess.run(["g++", "-O1", "-std=c++17", "-fsanitize=address", "-fno-omit-frame-pointer", str(src),
                    "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
    return r.stdout
