"""GPU parity of Ax / Atx (through the C ABI) against the golden vectors of
the reference's own code and against the oracle.  Tolerance: relative L2
error <= 1e-5 in FP32 (the spec bar); Atx additionally bit-exact
(same operation order per voxel as the reference)."""
import glob
import os

import numpy as np
import pytest

import asd_pocs_mex_cuda_demo_gb300 as pkg
from conftest import GOLDEN, rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5
PROJ = sorted(glob.glob(os.path.join(GOLDEN, "proj_*.npz")))


@pytest.mark.parametrize("path", PROJ, ids=[os.path.basename(p) for p in PROJ])
def test_mex_level_vs_reference_vectors(gpu, path):
    d = np.load(path)
    nx, ny, nz, na, nb = (int(v) for v in d["dims"])
    SO, OD, vx, det = d["geo"]
    for k, a in enumerate(d["angles"]):
        para = dict(SO=SO, OD=OD, vxlsize=vx, nx=nx, ny=ny, nz=nz, phi=-a / 180 * np.pi,
                    detsize=det, na=na, nb=nb)
        y, sr = pkg.Ax_cone_gpu(d["x"], para)
        assert rel_l2(y, d["y"][k]) <= TOL, (a, rel_l2(y, d["y"][k]))
        assert rel_l2(sr, d["sr"][k]) <= TOL
        b, sc = pkg.Atx_cone_gpu(d["yview"], para)
        assert np.array_equal(b, d["bp"][k]), (a, rel_l2(b, d["bp"][k]))
        assert np.array_equal(sc, d["sc"][k])


CASES = [
    # nx, ny, nz, na, nb, SO, OD, det
    (256, 256, 1, 512, 1, 541.0, 408.0, 1.0),
    (512, 512, 1, 888, 1, 541.0, 408.0, 1.0),
    (1, 1, 1, 3, 1, 541.0, 408.0, 1.0),
    (3, 17, 1, 1, 1, 541.0, 408.0, 1.0),
    (40, 40, 1, 80, 2, 405.941, 500.31, 0.6),
    (48, 40, 24, 96, 48, 1000.0, 500.0, 0.8 * 5),
    (17, 9, 5, 33, 7, 300.0, 200.0, 1.3),
    # cone beam with the magnification and bins per voxel of 256^3 on a 512^2
    # detector at 0.8 mm, SID 1000 / SDD 1500 mm
    (64, 64, 64, 128, 128, 1000.0, 500.0, 0.8 * 4),
]


@pytest.mark.parametrize("case", CASES, ids=[str(c[:5]) for c in CASES])
def test_launchers_vs_oracle(gpu, oracle_mod, case):
    nx, ny, nz, na, nb, SO, OD, det = case
    rng = np.random.default_rng(sum(case[:5]))
    vx = SO / (SO + OD) * det * na / nx
    x = rng.random(nx * ny * nz).astype(np.float32)
    yv = rng.standard_normal(na * nb).astype(np.float32)
    for a in [0.0, 90.0, 180.0, 270.0, 45.0] + rng.uniform(0, 360, 5).tolist():
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, det, na, nb)
        yo, so = oracle_mod.ax(x, g, nx, ny, nz)
        bo, co = oracle_mod.atx(yv, g, nx, ny, nz)
        y = np.zeros(na * nb, np.float32)
        sr = np.zeros(na * nb, np.float32)
        pkg.Ax_cone_mf_gpu_new(x, y, sr, g["cos_phi"], g["sin_phi"], g["y_det"], g["z_det"],
                               g["SO"], g["OD"], g["scale"], 1.0, nx, ny, nz, na, nb)
        b = np.zeros(nx * ny * nz, np.float32)
        sc = np.zeros(nx * ny * nz, np.float32)
        pkg.Atx_cone_mf_gpu_new(b, yv, sc, g["cos_phi"], g["sin_phi"], g["y_det"],
                                g["z_det"], g["SO"], g["OD"], g["scale"], g["det"],
                                g["det"], 1.0, nx, ny, nz, na, nb)
        assert rel_l2(y, yo) <= TOL, (a, rel_l2(y, yo))
        assert rel_l2(sr, so) <= TOL
        assert np.array_equal(b, bo), (a, rel_l2(b, bo))
        assert np.array_equal(sc, co)


@pytest.mark.parametrize("dims", [(48, 40, 1, 96, 1), (24, 20, 12, 48, 24)])
def test_atx_detector_off_grid(gpu, oracle_mod, dims):
    """Launcher callers may pass any detector coordinates; the backprojector
    then walks the reference's whole window (no shadow narrowing) and stays
    bit-identical."""
    nx, ny, nz, na, nb = dims
    SO, OD, det = 541.0, 408.0, 1.0
    rng = np.random.default_rng(nx * nz)
    vx = SO / (SO + OD) * det * na / nx
    yv = rng.standard_normal(na * nb).astype(np.float32)
    for a in (17.0, 133.0, 251.0):
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, det, na, nb)
        g["y_det"] = (g["y_det"] + rng.uniform(-0.3, 0.3, na) * g["det"]).astype(np.float32)
        if nb > 1:
            g["z_det"] = (g["z_det"] * 1.07).astype(np.float32)
        bo, co = oracle_mod.atx(yv, g, nx, ny, nz)
        b = np.zeros(nx * ny * nz, np.float32)
        sc = np.zeros(nx * ny * nz, np.float32)
        pkg.Atx_cone_mf_gpu_new(b, yv, sc, g["cos_phi"], g["sin_phi"], g["y_det"],
                                g["z_det"], g["SO"], g["OD"], g["scale"], g["det"],
                                g["det"], 1.0, nx, ny, nz, na, nb)
        assert np.array_equal(b, bo), (a, rel_l2(b, bo))
        assert np.array_equal(sc, co)


def test_device_pointer_variants(gpu, oracle_mod):
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    nx = ny = 96
    nz, na, nb = 1, 192, 1
    SO, OD, det = 541.0, 408.0, 1.0
    vx = SO / (SO + OD) * det * na / nx
    g = oracle_mod.gateway_geometry(-0.7, SO, OD, vx, det, na, nb)
    x = torch.rand(nx * ny * nz, device=gpu)
    ydet = torch.tensor(g["y_det"], device=gpu)
    zdet = torch.tensor(g["z_det"], device=gpu)
    y = torch.empty(na * nb, device=gpu)
    sr = torch.empty(na * nb, device=gpu)
    s = torch.cuda.current_stream().cuda_stream
    L = load()
    check(L.asdpocs_ax_device(x.data_ptr(), y.data_ptr(), sr.data_ptr(), g["cos_phi"],
                              g["sin_phi"], ydet.data_ptr(), zdet.data_ptr(), g["SO"],
                              g["OD"], g["scale"], 1.0, nx, ny, nz, na, nb, s))
    b = torch.empty_like(x)
    sc = torch.empty_like(x)
    check(L.asdpocs_atx_device(b.data_ptr(), y.data_ptr(), sc.data_ptr(), g["cos_phi"],
                               g["sin_phi"], ydet.data_ptr(), zdet.data_ptr(), g["SO"],
                               g["OD"], g["scale"], g["det"], g["det"], 1.0, nx, ny, nz,
                               na, nb, s))
    torch.cuda.synchronize()
    yo, so = oracle_mod.ax(x.cpu().numpy(), g, nx, ny, nz)
    assert rel_l2(y.cpu().numpy(), yo) <= TOL
    bo, co = oracle_mod.atx(y.cpu().numpy(), g, nx, ny, nz)
    assert np.array_equal(b.cpu().numpy(), bo) and np.array_equal(sc.cpu().numpy(), co)


def test_adjointness_gpu(gpu):
    n, na = 128, 256
    SO, OD, det = 541.0, 408.0, 1.0
    vx = SO / (SO + OD) * det * na / n
    rng = np.random.default_rng(11)
    x = rng.random(n * n).astype(np.float32)
    yv = rng.random(na).astype(np.float32)
    for a in (13.0, 77.0, 200.0):
        para = dict(SO=SO, OD=OD, vxlsize=vx, nx=n, ny=n, nz=1, phi=-a / 180 * np.pi,
                    detsize=det, na=na, nb=1)
        Ax, _ = pkg.Ax_cone_gpu(x, para)
        Aty, _ = pkg.Atx_cone_gpu(yv, para)
        lhs = float(np.dot(Ax.astype(np.float64), yv))
        rhs = float(np.dot(x.astype(np.float64), Aty))
        assert abs(lhs - rhs) / abs(lhs) < 2e-5


def test_atx_non_finite_view_values_propagate_like_reference(gpu, oracle_mod):
    # a NaN / inf view value reaches every voxel whose footprint window holds
    # its bin, through the zero chords too (0*NaN), as in the reference loop
    n, na = 64, 128
    SO, OD, det = 541.0, 408.0, 1.0
    vx = SO / (SO + OD) * det * na / n
    yv = np.random.default_rng(5).random(na).astype(np.float32)
    yv[40] = np.nan
    yv[90] = np.inf
    for a in (0.0, 33.0, 90.0):
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, det, na, 1)
        bo, co = oracle_mod.atx(yv, g, n, n, 1)
        para = dict(SO=SO, OD=OD, vxlsize=vx, nx=n, ny=n, nz=1, phi=-a / 180 * np.pi,
                    detsize=det, na=na, nb=1)
        b, sc = pkg.Atx_cone_gpu(yv, para)
        assert np.isnan(bo).any()
        assert np.array_equal(b, bo, equal_nan=True), a
        assert np.array_equal(sc, co)


@pytest.mark.parametrize("angle", [0.0, 90.0, 180.0, 270.0])
def test_axis_parallel_central_ray(gpu, oracle_mod, angle):
    # with an odd detector the central bin's ray is axis-parallel at these
    # angles; the reference's chord then ignores one coordinate (length 1 for
    # every voxel of the footprint window)
    nx, ny, na = 33, 17, 41
    SO, OD, det = 541.0, 408.0, 1.0
    vx = SO / (SO + OD) * det * na / nx
    yv = np.random.default_rng(9).random(na).astype(np.float32)
    g = oracle_mod.gateway_geometry(-angle / 180 * np.pi, SO, OD, vx, det, na, 1)
    bo, co = oracle_mod.atx(yv, g, nx, ny, 1)
    para = dict(SO=SO, OD=OD, vxlsize=vx, nx=nx, ny=ny, nz=1, phi=-angle / 180 * np.pi,
                detsize=det, na=na, nb=1)
    b, sc = pkg.Atx_cone_gpu(yv, para)
    assert np.array_equal(b, bo) and np.array_equal(sc, co)


@pytest.mark.parametrize("dims", [(128, 128, 1, 256, 1), (48, 40, 24, 64, 48)])
def test_adjoint_check_on_gpu(gpu, dims):
    """<Ax, y> and <x, A^T y> accumulated in FP64 on the GPU agree, and match
    the host FP64 dots of the GPU projections.  In 2-D the reference's
    forward march and backprojector use the same exact intersection lengths
    (agreement to FP32 rounding); in 3-D its forward march approximates
    them (a piecewise column march against find_l_3d's exact chords), so
    the pair is adjoint to about 1e-4 only."""
    nx, ny, nz, na, nb = dims
    SO, OD, det = 541.0, 408.0, 1.0
    vx = SO / (SO + OD) * det * na / max(nx, ny)
    rng = np.random.default_rng(nz)
    x = rng.random(nx * ny * nz).astype(np.float32)
    yv = rng.random(na * nb).astype(np.float32)
    for a in (13.0, 200.0):
        para = dict(SO=SO, OD=OD, vxlsize=vx, nx=nx, ny=ny, nz=nz, phi=-a / 180 * np.pi,
                    detsize=det, na=na, nb=nb)
        lhs, rhs = pkg.adjoint_check(x, yv, para)
        assert abs(lhs - rhs) / abs(lhs) < (2e-5 if nz == 1 else 5e-4)
        Ax, _ = pkg.Ax_cone_gpu(x, para)
        Aty, _ = pkg.Atx_cone_gpu(yv, para)
        assert abs(lhs - float(np.dot(Ax.astype(np.float64), yv))) <= 1e-9 * abs(lhs)
        assert abs(rhs - float(np.dot(x.astype(np.float64), Aty))) <= 1e-9 * abs(rhs)


def _launch_pair(g, x, yv, nx, ny, nz, na, nb):
    y = np.zeros(na * nb, np.float32)
    sr = np.zeros(na * nb, np.float32)
    pkg.Ax_cone_mf_gpu_new(x, y, sr, g["cos_phi"], g["sin_phi"], g["y_det"], g["z_det"],
                           g["SO"], g["OD"], g["scale"], 1.0, nx, ny, nz, na, nb)
    b = np.zeros(nx * ny * nz, np.float32)
    sc = np.zeros(nx * ny * nz, np.float32)
    pkg.Atx_cone_mf_gpu_new(b, yv, sc, g["cos_phi"], g["sin_phi"], g["y_det"], g["z_det"],
                            g["SO"], g["OD"], g["scale"], g["det"], g["det"], 1.0, nx, ny,
                            nz, na, nb)
    return y, sr, b, sc


def test_cone_beam_full_size_views(gpu, oracle_mod):
    """Two views of the full cone-beam workload's geometry -- a 256^3 volume of
    1 mm voxels, a 512 x 512 detector at 0.8 mm, SID 1000 / SDD 1500 mm --
    through the launcher symbols: Ax within 1e-5 of the oracle, Atx (the
    z-column backward step) bit for bit."""
    n, na = 256, 512
    SO, OD, det, vx = 1000.0, 500.0, 0.8, 1.0
    rng = np.random.default_rng(256)
    x = rng.random(n ** 3).astype(np.float32)
    yv = rng.standard_normal(na * na).astype(np.float32)
    for a in (17.0, 123.0):
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, det, na, na)
        y, sr, b, sc = _launch_pair(g, x, yv, n, n, n, na, na)
        yo, so = oracle_mod.ax(x, g, n, n, n)
        assert rel_l2(y, yo) <= TOL, (a, rel_l2(y, yo))
        assert rel_l2(sr, so) <= TOL
        bo, co = oracle_mod.atx(yv, g, n, n, n)
        assert np.array_equal(b, bo), (a, rel_l2(b, bo), int((b != bo).sum()))
        assert np.array_equal(sc, co)


@pytest.mark.parametrize("angle", [0.0, 17.0, 45.0, 123.0, 250.0])
def test_fan_beam_ax_against_fp64_siddon(gpu, oracle_mod, angle):
    """In 2-D the reference's column march is exact: the GPU forward step's
    sums and ray lengths equal the FP64 Siddon projector's (exact
    intersection lengths accumulated in double) to FP32 rounding, on the
    512^2 / 888-bin fan-beam geometry."""
    n, na = 512, 888
    SO, OD, det = 541.0, 408.0, 1.0
    vx = SO / (SO + OD) * det * na / n
    x = np.random.default_rng(int(angle)).random(n * n).astype(np.float32)
    g = oracle_mod.gateway_geometry(-angle / 180 * np.pi, SO, OD, vx, det, na, 1)
    y, sr, _, _ = _launch_pair(g, x, np.zeros(na, np.float32), n, n, 1, na, 1)
    ye, sre = oracle_mod.siddon_ax(x, g, n, n, 1)
    assert rel_l2(y, ye) <= 5e-6, rel_l2(y, ye)
    assert rel_l2(sr, sre) <= 5e-6, rel_l2(sr, sre)


@pytest.mark.parametrize("case", [(512, 512, 1, 888, 1, 541.0, 408.0, 1.0),
                                  (64, 64, 64, 128, 128, 1000.0, 500.0, 0.8 * 4),
                                  (96, 80, 40, 192, 96, 1000.0, 500.0, 0.8 * 256 / 96),
                                  (17, 9, 5, 33, 7, 300.0, 200.0, 1.3)],
                         ids=lambda c: str(c[:5]))
def test_exact_forward_mode_against_fp64_siddon(gpu, oracle_mod, case):
    """The exact forward projection (asdpocs_ax_siddon: FP64 crossing
    parameters, FP32 lengths and sums) against the FP64 Siddon oracle within
    1e-5, in 2-D and 3-D.  The reference's own 3-D column march deviates from
    the same oracle by about 1e-3 (its split fractions are measured from one
    column end); in 2-D both are exact."""
    nx, ny, nz, na, nb, SO, OD, det = case
    rng = np.random.default_rng(nx + nz)
    vx = SO / (SO + OD) * det * na / nx
    x = rng.random(nx * ny * nz).astype(np.float32)
    worst_march = 0.0
    for a in (0.0, 33.0, 90.0, 137.0):
        g = oracle_mod.gateway_geometry(-a / 180 * np.pi, SO, OD, vx, det, na, nb)
        ye, se = oracle_mod.siddon_ax(x, g, nx, ny, nz)
        y = np.zeros(na * nb, np.float32)
        sr = np.zeros(na * nb, np.float32)
        pkg.Ax_siddon_mf_gpu(x, y, sr, g["cos_phi"], g["sin_phi"], g["y_det"], g["z_det"],
                             g["SO"], g["OD"], g["scale"], 1.0, nx, ny, nz, na, nb)
        assert rel_l2(y, ye) <= TOL, (a, rel_l2(y, ye))
        assert rel_l2(sr, se) <= TOL, (a, rel_l2(sr, se))
        ym, _, _, _ = _launch_pair(g, x, np.zeros(na * nb, np.float32), nx, ny, nz, na, nb)
        worst_march = max(worst_march, rel_l2(ym, ye))
    if nz > 8:
        assert worst_march > 1e-4  # the reference march's documented 3-D deviation


@pytest.mark.parametrize("dims", [(512, 512, 1, 888, 1), (65, 31, 1, 97, 1), (40, 24, 1, 57, 3),
                                  (9, 7, 5, 19, 11)])
def test_chained_device_projections_wait_for_each_other(gpu, oracle_mod, dims):
    """Ax then Atx then Ax ..., each on the previous one's output and on
    detector coordinates that a copy just before it wrote, without a
    synchronisation in between (each kernel starts while the one before it
    drains), captured in a graph as well: the same bits as with one."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    nx, ny, nz, na, nb = dims
    L, N, M = load(), nx * ny * nz, na * nb
    geo = [oracle_mod.gateway_geometry(-a / 180 * np.pi, 541.0, 408.0, 541.0 / 949.0 * na / nx,
                                       1.0, na, nb) for a in (0.0, 31.0, 90.0, 211.0)]
    yd = [torch.from_numpy(np.ascontiguousarray(g["y_det"], np.float32)).cuda() for g in geo]
    zd = [torch.from_numpy(np.ascontiguousarray(g["z_det"], np.float32)).cuda() for g in geo]
    x0 = torch.from_numpy(np.random.default_rng(3).random(N).astype(np.float32)).cuda()
    x, sc = torch.empty(N, device="cuda"), torch.empty(N, device="cuda")
    y, sr = torch.empty(M, device="cuda"), torch.empty(M, device="cuda")
    py, pz = torch.empty(na, device="cuda"), torch.empty(nb, device="cuda")

    def chain(sync):
        st = torch.cuda.current_stream().cuda_stream
        x.copy_(x0)
        for _ in range(3):
            for g, a, b in zip(geo, yd, zd):
                view = (g["cos_phi"], g["sin_phi"], py.data_ptr(), pz.data_ptr(), g["SO"],
                        g["OD"], g["scale"])
                py.fill_(float("nan"))
                torch.add(a, 0.0, out=py)
                torch.add(b, 0.0, out=pz)
                check(L.asdpocs_ax_device(x.data_ptr(), y.data_ptr(), sr.data_ptr(), *view,
                                          1.0, *dims, st))
                if sync:
                    torch.cuda.synchronize()
                check(L.asdpocs_atx_device(x.data_ptr(), y.data_ptr(), sc.data_ptr(), *view,
                                           g["det"], g["det"], 1.0, *dims, st))
                if sync:
                    torch.cuda.synchronize()
                x.div_(x.abs().max())
        return x.clone()

    want = chain(True)
    assert torch.isfinite(want).all() and want.abs().max() == 1
    assert torch.equal(chain(False), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain(False)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_small_host_calls_equal_large_ones(gpu, oracle_mod):
    """Calls with few bytes of arguments pass them through page-locked memory
    (up to 512 KiB of inputs, 256 KiB of results): on both sides of the
    limits, and from several threads at once, the bits of the device entry
    points."""
    import threading

    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    L = load()
    dims = [(8, 8, 1, 9, 1), (128, 256, 1, 64, 1), (129, 256, 1, 64, 1), (361, 362, 1, 64, 1),
            (363, 362, 1, 64, 1), (20, 24, 30, 200, 300), (20, 24, 30, 400, 330)]
    jobs = []
    for k, (nx, ny, nz, na, nb) in enumerate(dims):
        rng = np.random.default_rng(k)
        para = dict(SO=541.0, OD=408.0, vxlsize=541.0 / 949.0 * na / nx, nx=nx, ny=ny, nz=nz,
                    phi=-0.3 - k, detsize=1.0, na=na, nb=nb)
        g = oracle_mod.gateway_geometry(para["phi"], 541.0, 408.0, para["vxlsize"], 1.0, na, nb)
        x = rng.random(nx * ny * nz).astype(np.float32)
        y = rng.random(na * nb).astype(np.float32)
        dev = [torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
               for a in (x, y, g["y_det"], g["z_det"])]
        out = [torch.empty(n, device="cuda") for n in (y.size, y.size, x.size, x.size)]
        st = torch.cuda.current_stream().cuda_stream
        view = (g["cos_phi"], g["sin_phi"], dev[2].data_ptr(), dev[3].data_ptr(), g["SO"],
                g["OD"], g["scale"])
        check(L.asdpocs_ax_device(dev[0].data_ptr(), out[0].data_ptr(), out[1].data_ptr(), *view,
                                  1.0, nx, ny, nz, na, nb, st))
        check(L.asdpocs_atx_device(out[2].data_ptr(), dev[1].data_ptr(), out[3].data_ptr(), *view,
                                   g["det"], g["det"], 1.0, nx, ny, nz, na, nb, st))
        torch.cuda.synchronize()
        jobs.append((para, x, y, [o.cpu().numpy() for o in out]))

    wrong = []

    def work(order):
        for k in order:
            para, x, y, want = jobs[k]
            got = pkg.Ax_cone_gpu(x, para) + pkg.Atx_cone_gpu(y, para)
            if not all(np.array_equal(a, b) for a, b in zip(got, want)):
                wrong.append(dims[k])

    work(range(len(jobs)))
    threads = [threading.Thread(target=work, args=(np.roll(range(len(jobs)), t),))
               for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_back_projection_waits_for_the_detector_rows(gpu, oracle_mod):
    """A fan-beam Atx whose detector row lies where the kernel before it, which
    lets its successor start early, writes it: 0, where the planar form holds,
    and other heights in turn, the bits of synchronised calls."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    n, na, L = 64, 128, load()
    g = oracle_mod.gateway_geometry(-0.4, 541.0, 408.0, 541.0 / 949.0 * na / n, 1.0, na, 1)
    y = torch.rand(na, device="cuda")
    yd = torch.from_numpy(np.ascontiguousarray(g["y_det"], np.float32)).cuda()
    # one ray along a row of 8192 voxels: their sum goes to the detector row
    long = [torch.full((8192,), v, device="cuda") for v in (0.0, 1e-4, 0.0, 2e-4, 3e-4)]
    zero, row, sr = (torch.zeros(1, device="cuda") for _ in range(3))

    def run(sync):
        st, out = torch.cuda.current_stream().cuda_stream, []
        for k in range(20):
            x, sc = torch.empty(n * n, device="cuda"), torch.empty(n * n, device="cuda")
            check(L.asdpocs_ax_device(long[k % 5].data_ptr(), row.data_ptr(), sr.data_ptr(), 1.0,
                                      0.0, zero.data_ptr(), zero.data_ptr(), 9000.0, 9000.0, 1.0,
                                      1.0, 8192, 1, 1, 1, 1, st))
            if sync:
                torch.cuda.synchronize()
            check(L.asdpocs_atx_device(x.data_ptr(), y.data_ptr(), sc.data_ptr(), g["cos_phi"],
                                       g["sin_phi"], yd.data_ptr(), row.data_ptr(), g["SO"],
                                       g["OD"], g["scale"], g["det"], g["det"], 1.0, n, n, 1, na,
                                       1, st))
            if sync:
                torch.cuda.synchronize()
            out += [x, sc, row.clone()]
        torch.cuda.synchronize()
        return out

    want = run(True)
    assert len({float(r) for r in want[2::3]}) == 4
    assert not torch.equal(want[0], want[3])  # the height matters
    for a, b in zip(run(False), want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dims", [(32, 32, 1, 64, 1), (16, 16, 8, 32, 16), (96, 96, 96, 160, 160)])
def test_back_projection_leaves_the_callers_error(gpu, oracle_mod, dims):
    """An error of a call of the caller's own that it has not yet read (here a
    device number that does not exist) is still there after asdpocs_atx_device."""
    import ctypes

    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    nx, ny, nz, na, nb = dims
    rt = ctypes.CDLL("libcudart.so.13")  # the one the library is linked to
    g = oracle_mod.gateway_geometry(-0.4, 541.0, 408.0, 541.0 / 949.0 * na / nx, 1.0, na, nb)
    x, sc = torch.empty(nx * ny * nz, device="cuda"), torch.empty(nx * ny * nz, device="cuda")
    y = torch.rand(na * nb, device="cuda")
    yd, zd = (torch.from_numpy(np.ascontiguousarray(g[k], np.float32)).cuda()
              for k in ("y_det", "z_det"))
    st = torch.cuda.current_stream().cuda_stream

    def call():
        check(load().asdpocs_atx_device(x.data_ptr(), y.data_ptr(), sc.data_ptr(), g["cos_phi"],
                                        g["sin_phi"], yd.data_ptr(), zd.data_ptr(), g["SO"],
                                        g["OD"], g["scale"], g["det"], g["det"], 1.0, *dims, st))

    call()
    torch.cuda.synchronize()
    want, err = (x.clone(), sc.clone()), rt.cudaSetDevice(9999)
    assert err != 0
    try:
        call()
        assert rt.cudaPeekAtLastError() == err
    finally:
        rt.cudaGetLastError()
    torch.cuda.synchronize()
    assert torch.equal(x, want[0]) and torch.equal(sc, want[1])


def test_back_projection_beside_another_threads_capture(gpu, oracle_mod):
    """asdpocs_atx_device on one thread, with the scratch of its z-column form,
    while another thread captures a stream of its own: the capture stays valid,
    and the results are those of a call alone."""
    import threading

    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    n, na = 96, 160
    N = n ** 3
    g = oracle_mod.gateway_geometry(-0.4, 541.0, 408.0, 541.0 / 949.0 * na / n, 1.0, na, na)
    y = torch.rand(na * na, device="cuda")
    yd, zd = (torch.from_numpy(np.ascontiguousarray(g[k], np.float32)).cuda()
              for k in ("y_det", "z_det"))
    out = [torch.empty(N, device="cuda") for _ in range(4)]
    a = torch.ones(1000, device="cuda")
    other, errors = torch.cuda.Stream(), []
    torch.cuda.synchronize()

    def call(x, sc):
        try:
            check(load().asdpocs_atx_device(x.data_ptr(), y.data_ptr(), sc.data_ptr(),
                                            g["cos_phi"], g["sin_phi"], yd.data_ptr(),
                                            zd.data_ptr(), g["SO"], g["OD"], g["scale"], g["det"],
                                            g["det"], 1.0, n, n, n, na, na, other.cuda_stream))
        except Exception as e:  # the test reports it
            errors.append(e)

    call(out[0], out[1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        a.mul_(2.0)
        for _ in range(2):
            t = threading.Thread(target=call, args=(out[2], out[3]))
            t.start()
            t.join()
        call(out[2], out[3])  # and on the capturing thread
        a.add_(1.0)
    graph.replay()
    torch.cuda.synchronize()
    assert not errors
    assert float(a[0]) == 3.0
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])


@pytest.mark.parametrize("na", [900, 1100, 4096])
def test_back_projection_on_fine_detectors(gpu, oracle_mod, na):
    """A 64^2 image on 14, 17 and 64 bins a voxel: blocks that stage their rays,
    blocks that see more than they can stage, and both launch shapes."""
    n = 64
    y = np.random.default_rng(na).standard_normal(na).astype(np.float32)
    for a in (0.3, 45.0, 200.0):
        para = dict(SO=9000.0, OD=5000.0, vxlsize=9.0 / 14.0 * na / n, nx=n, ny=n, nz=1, na=na,
                    nb=1, phi=-a / 180 * np.pi, detsize=1.0)
        g = oracle_mod.gateway_geometry(para["phi"], 9000.0, 5000.0, para["vxlsize"], 1.0, na, 1)
        bo, co = oracle_mod.atx(y, g, n, n, 1)
        b, c = pkg.Atx_cone_gpu(y, para)
        assert np.array_equal(b, bo) and np.array_equal(c, co), a


@pytest.mark.parametrize("dims", [(24, 20, 12, 137, 37), (40, 33, 17, 500, 9), (17, 40, 40, 64, 83)])
def test_rays_by_rows_equal_rays_alone(gpu, oracle_mod, dims):
    """A cone-beam Ax of few rays has a warp per ray, of many a warp for four rows
    of a detector column: a detector's rows give the same bits when more rows lie
    above them."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    nx, ny, nz, na, nb = dims
    more = nb + 5500 // na + 2
    assert na * nb < 5472 < na * more
    x = torch.rand(nx * ny * nz, device="cuda", generator=torch.Generator("cuda").manual_seed(na))
    g = oracle_mod.gateway_geometry(-0.7, 541.0, 408.0, 541.0 / 949.0 * na / max(nx, ny), 1.0, na,
                                    more)
    yd, zd = (torch.from_numpy(np.ascontiguousarray(g[k], np.float32)).cuda()
              for k in ("y_det", "z_det"))
    zd = zd.roll(-(more - nb) // 2).contiguous()  # the few rows near the middle
    st = torch.cuda.current_stream().cuda_stream
    out = []
    for rows in (nb, more):
        y, sr = torch.empty(na * rows, device="cuda"), torch.empty(na * rows, device="cuda")
        check(load().asdpocs_ax_device(x.data_ptr(), y.data_ptr(), sr.data_ptr(), g["cos_phi"],
                                       g["sin_phi"], yd.data_ptr(), zd.data_ptr(), g["SO"],
                                       g["OD"], g["scale"], 1.0, nx, ny, nz, na, rows, st))
        out.append((y[:na * nb], sr[:na * nb]))
    assert float(out[0][1].max()) > 0
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def test_refused_launches_leave_no_error_behind(gpu):
    """A launch that CUDA refuses (an image of 65536 tile rows) is reported by its
    own call; the next calls, which ask CUDA for its last error, work."""
    import ctypes

    import torch

    from asd_pocs_mex_cuda_demo_gb300 import phantoms
    from asd_pocs_mex_cuda_demo_gb300._lib import AsdpocsError, check, load

    rt = ctypes.CDLL("libcudart.so.13")
    nx, ny, na = 8, 8 * 65536, 16
    x, sc = torch.empty(nx * ny, device="cuda"), torch.empty(nx * ny, device="cuda")
    y, yd, zd = (torch.rand(n, device="cuda") for n in (na, na, 1))
    with pytest.raises(AsdpocsError, match="invalid"):
        check(load().asdpocs_atx_device(x.data_ptr(), y.data_ptr(), sc.data_ptr(), 1.0, 0.0,
                                        yd.data_ptr(), zd.data_ptr(), 4000.0, 2000.0, 1.0, 1.0,
                                        1.0, 1.0, nx, ny, 1, na, 1,
                                        torch.cuda.current_stream().cuda_stream))
    assert rt.cudaPeekAtLastError() == 0
    para = dict(SO=541.0, OD=408.0, vxlsize=1.0, nx=16, ny=16, nz=1, na=32, nb=1, detsize=1.0,
                phi_vec=phantoms.views(3), maxnumIter=1, numOfgradients=1)
    pkg.ASD_POCS_cuda(np.random.default_rng(0).random((32, 3)), para)


def test_back_projection_refuses_volumes_beyond_a_launch(gpu):
    """A volume of more than 65535 tile rows (ceil(ny / 8) * nz) is refused whichever
    form its size would take, in a capture or not; one within them is not."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import AsdpocsError, check, load

    nx, ny, na, nb = 16, 2048, 64, 64
    x, sc = torch.empty(nx * ny * 300, device="cuda"), torch.empty(nx * ny * 300, device="cuda")
    y, yd = torch.rand(na * nb, device="cuda"), torch.arange(na, device="cuda") * 64.0 - 2016.0

    def call(nz):
        check(load().asdpocs_atx_device(x.data_ptr(), y.data_ptr(), sc.data_ptr(), 1.0, 0.0,
                                        yd.data_ptr(), yd.data_ptr(), 4000.0, 2000.0, 1.0, 64.0,
                                        64.0, 1.0, nx, ny, nz, na, nb,
                                        torch.cuda.current_stream().cuda_stream))

    call(255)
    for nz in (256, 300):
        with pytest.raises(AsdpocsError, match="invalid"):
            call(nz)
    torch.cuda.synchronize()
