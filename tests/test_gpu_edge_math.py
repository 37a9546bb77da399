"""The FP32 mode's own edge arithmetic (cutoff function, edge length) is no further
from 64 bits than the CUDA functions it stands for, sincospif, sqrtf and the
division: largest and rms errors over every float of the ranges, both measured in
one sweep on the GPU (tests/cpp/edge_math.cu)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sweep(tmp_path_factory):
    out = tmp_path_factory.mktemp("edge") / "libedge_math.so"
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-Xcompiler", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "dmg-md_b200", "csrc"), "-o", str(out),
                    os.path.join(ROOT, "tests", "cpp", "edge_math.cu")], check=True)
    lib = ctypes.CDLL(str(out))

    def run(which, lo, hi):
        first, last = (int(np.float32(v).view(np.uint32)) for v in (lo, hi))
        n = (last - first) // 32 * 32
        acc = np.zeros(12)
        assert lib.edge_math(which, ctypes.c_uint(first), ctypes.c_uint(n),
                             acc.ctypes.data_as(ctypes.c_void_p)) == 0
        return acc[0::2], np.sqrt(acc[1::2] / n)      # largest, rms
    return run


# d / rc: the whole range, and the tail where fc vanishes
@pytest.mark.parametrize("lo,hi", [(2.0 ** -10, 1.0), (0.9, 1.0)])
def test_cutoff_function(sweep, lo, hi):
    largest, rms = sweep(0, lo, hi)
    fc, fc_cuda, slope, slope_cuda, rel, rel_cuda = range(6)
    assert largest[fc] <= largest[fc_cuda] and rms[fc] <= rms[fc_cuda]
    assert largest[slope] <= largest[slope_cuda] and rms[slope] <= rms[slope_cuda]
    assert rms[rel] <= rms[rel_cuda]


# d^2 in A^2: two binades have every mantissa of a root; short, usual and long edges
@pytest.mark.parametrize("lo", [2.0 ** -20, 1.0, 16.0])
def test_edge_length(sweep, lo):
    largest, rms = sweep(1, lo, 4.0 * lo)
    assert largest[4] == 0.0                                   # d is sqrtf's everywhere
    assert largest[2] <= largest[3] and rms[2] <= rms[3] * (1.0 + 1e-6)
