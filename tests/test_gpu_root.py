"""The cone-beam backward step's square root (root_rn) against the IEEE one,
on the GPU, for every float from its lower limit to 2^40: the same bits."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_root_is_correctly_rounded(gpu):
    src = os.path.join(ROOT, "tests", "device_math", "root_gpu.cu")
    out = os.path.join(ROOT, "tests", "device_math", "_build", "libroot_gpu.so")
    os.makedirs(os.path.dirname(out), exist_ok=True)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-O3", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a",
                    "-fmad=false", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC",
                    "-o", out, src], check=True)
    L = C.CDLL(out)
    L.root_mismatches.restype = C.c_longlong
    L.root_mismatches.argtypes = [C.c_uint, C.c_uint]
    L.root_min.restype = C.c_float
    lo = int(np.float32(L.root_min()).view(np.uint32))
    hi = int(np.float32(2.0 ** 40).view(np.uint32))
    assert L.root_mismatches(lo, hi) == 0
