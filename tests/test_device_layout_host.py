"""Rows of a detector column projected together, and the 2-D chord table's
layout (csrc/projector.cuh), built for the host."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT, rel_l2

SRC = os.path.join(ROOT, "tests", "device_math", "dm_layout.cu")
SO_PATH = os.path.join(ROOT, "tests", "device_math", "_build", "libdm_layout.so")
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
    L.dm_ax_rows.argtypes = [F, F, F, C.c_float, C.c_float, F, F] + [C.c_float] * 4 + [C.c_int] * 6
    L.dm_atx_chords.argtypes = [F, F, F, C.c_float, C.c_float, F] + [C.c_float] * 4 + [C.c_int] * 3
    return L


def _p(a):
    return a.ctypes.data_as(F)


@pytest.mark.parametrize("case", [(24, 20, 12, 48, 24, 1000.0, 500.0, 3.2),
                                  (13, 11, 7, 27, 9, 300.0, 200.0, 1.3),
                                  (31, 33, 9, 60, 21, 1000.0, 500.0, 6.0),
                                  (40, 9, 33, 30, 6, 300.0, 200.0, 2.0)],
                         ids=lambda c: str(c[:5]))
def test_rows_together_equal_rays_alone(dm, oracle_mod, case):
    nx, ny, nz, na, nb, SO, OD, det = case
    rng = np.random.default_rng(nx)
    vx = SO / (SO + OD) * det * na / max(nx, ny)
    x = rng.random(nx * ny * nz).astype(np.float32)
    for a in [0.0, 45.0, 90.0, 200.0] + rng.uniform(0, 360, 4).tolist():
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, det, na, nb)
        yd, zd = g["y_det"].copy(), g["z_det"].copy()
        out = []
        for rows in (0, 1):
            y, sr = np.zeros(na * nb, np.float32), np.zeros(na * nb, np.float32)
            dm.dm_ax_rows(_p(x), _p(y), _p(sr), g["cos_phi"], g["sin_phi"], _p(yd), _p(zd),
                          g["SO"], g["OD"], g["scale"], 1.0, nx, ny, nz, na, nb, rows)
            out.append((y, sr))
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1]), a
        yo, so = oracle_mod.ax(x, g, nx, ny, nz)
        assert rel_l2(out[1][0], yo) < 1e-6 and rel_l2(out[1][1], so) < 1e-6, a


@pytest.mark.parametrize("dims", [(64, 64, 128), (17, 23, 41), (50, 31, 77), (9, 8, 60)])
def test_chord_table_words(dm, oracle_mod, dims):
    """Heads in pairs, chords in planes of two per voxel: filled and read back, the
    table gives the oracle's Atx and chord sums bit for bit."""
    nx, ny, na = dims
    SO, OD, det = 541.0, 408.0, 1.0
    vx = SO / (SO + OD) * det * na / nx
    yv = np.random.default_rng(na).standard_normal(na).astype(np.float32)
    tables = 0
    for a in (0.0, 30.0, 45.0, 90.0, 200.0, 333.3):
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, det, na, 1)
        yd = g["y_det"].copy()
        b, sc = np.zeros(nx * ny, np.float32), np.zeros(nx * ny, np.float32)
        K = dm.dm_atx_chords(_p(b), _p(yv), _p(sc), g["cos_phi"], g["sin_phi"], _p(yd), g["SO"],
                             g["OD"], g["scale"], g["det"], nx, ny, na)
        if K == -1:  # the central ray of an odd detector
            assert na % 2 == 1 and a in (0.0, 90.0)
            continue
        tables += 1
        assert K >= 2 and K % 2 == 0
        bo, co = oracle_mod.atx(yv, g, nx, ny, 1)
        assert np.array_equal(b, bo) and np.array_equal(sc, co), a
    assert tables >= 4
