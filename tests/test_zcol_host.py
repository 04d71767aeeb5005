"""The z-column backward step's ray reads and sums (csrc/projector.cuh), built
for the host: volumes of few slices, whose warps hold two or four voxel columns
(16 or 8 lanes each), at views where some of a warp's columns lie outside the
detector and others do not."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = os.path.join(ROOT, "tests", "device_math", "dm_zcol.cu")
SO_PATH = os.path.join(ROOT, "tests", "device_math", "_build", "libdm_zcol.so")
HEADER = os.path.join(ROOT, "asd_pocs_mex_cuda_demo_gb300", "csrc", "projector.cuh")
F = C.POINTER(C.c_float)


@pytest.fixture(scope="module")
def dm():
    os.makedirs(os.path.dirname(SO_PATH), exist_ok=True)
    if not os.path.exists(SO_PATH) or any(
            os.path.getmtime(p) > os.path.getmtime(SO_PATH) for p in (SRC, HEADER)):
        subprocess.run(["nvcc", "-O2", "-std=c++17", "-shared", "-Xcompiler",
                        "-fPIC,-ffp-contract=off", "-o", SO_PATH, SRC], check=True)
    L = C.CDLL(SO_PATH)
    L.dm_zcol_walk.argtypes = [F, F, F, C.c_float, C.c_float, F, F] + [C.c_float] * 6 + [C.c_int] * 6
    L.dm_zcol_walk.restype = C.c_longlong
    return L


def _p(a):
    return a.ctypes.data_as(F) if a is not None else None


def walk(dm, g, y, nx, ny, nz, na, nb, lanes):
    x = np.zeros(nx * ny * nz, np.float32) if y is not None else None
    sc = np.zeros(nx * ny * nz, np.float32) if y is not None else None
    yd, zd = (np.ascontiguousarray(g[k], np.float32) for k in ("y_det", "z_det"))
    bad = dm.dm_zcol_walk(_p(x), _p(y), _p(sc), g["cos_phi"], g["sin_phi"], _p(yd), _p(zd),
                          g["SO"], g["OD"], g["scale"], g["det"], g["det"], 1.0, nx, ny, nz, na,
                          nb, lanes)
    return bad, x, sc


# nx, ny, nz, na, nb, SO, OD, lanes of a column, part of the fan the image fills
FULL = [(128, 128, 72, 257, 200, 541.0, 408.0, 8, 1.0), (160, 160, 48, 400, 120, 541.0, 408.0, 16, 1.0),
        (64, 64, 40, 48, 40, 100.0, 50.0, 8, 1.6), (48, 48, 9, 120, 30, 60.0, 60.0, 16, 1.7),
        (24, 24, 40, 40, 120, 20.0, 10.0, 8, 1.0), (40, 40, 16, 30, 1, 541.0, 408.0, 8, 1.0),
        (60, 50, 90, 100, 17, 400.0, 300.0, 16, 1.2), (50, 60, 3, 100, 3, 400.0, 300.0, 4, 1.0)]


@pytest.mark.parametrize("case", FULL, ids=lambda c: str(c[:5]) + f"-{c[7]}")
def test_reads_stay_within_the_padded_tables(dm, oracle_mod, case):
    nx, ny, nz, na, nb, SO, OD, lanes, fill = case
    vx = SO / (SO + OD) * na / nx * fill
    views = 0
    for a in np.arange(60) * 6.0 + (0.0 if na % 2 == 0 else 1.5):
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, 1.0, na, nb)
        bad, _, _ = walk(dm, g, None, nx, ny, nz, na, nb, lanes)
        if bad == -1:  # an axis-parallel ray
            continue
        views += 1
        assert bad == 0, (a, bad)
    assert views >= 50


@pytest.mark.parametrize("case", FULL[2:], ids=lambda c: str(c[:5]) + f"-{c[7]}")
@pytest.mark.parametrize("angle", [3.0, 45.0, 135.0, 201.3])
def test_sums_are_the_oracle_s(dm, oracle_mod, case, angle):
    """Bit for bit, whatever the lanes without pairs read."""
    nx, ny, nz, na, nb, SO, OD, lanes, fill = case
    vx = SO / (SO + OD) * na / nx * fill
    y = np.random.default_rng(na).standard_normal(na * nb).astype(np.float32)
    g = oracle_mod.gateway_geometry(-angle / 180 * np.pi, SO, OD, vx, 1.0, na, nb)
    bo, co = oracle_mod.atx(y, g, nx, ny, nz)
    bad, x, sc = walk(dm, g, y, nx, ny, nz, na, nb, lanes)
    assert bad == 0
    assert np.array_equal(x, bo) and np.array_equal(sc, co)
