"""The cone-beam backward step in voxel columns against its per-voxel form,
bit for bit, over the sizes and geometries where its lane and block layout and
its pair paths change: calls on host arrays take columns; asdpocs_atx_device
takes the per-voxel form for small volumes and while its stream is captured, so
one call is made plainly, one in a graph and one on host arrays."""
import ctypes as C

import numpy as np
import pytest

import asd_pocs_mex_cuda_demo_gb300 as pkg
from asd_pocs_mex_cuda_demo_gb300._lib import check, load

pytestmark = pytest.mark.gpu

# nx, ny, nz, na, nb, SO, OD (voxels), detector pitch (voxels), dz
CASES = [
    (20, 20, 20, 40, 30, 90.0, 45.0, 0.9, 1.0),       # 8 columns a block
    (41, 37, 33, 64, 70, 90.0, 45.0, 0.9, 1.0),       # ragged, one slice past a warp
    (40, 640, 10, 900, 24, 900.0, 450.0, 1.1, 1.0),   # 32 columns, 16 lanes
    (33, 1300, 7, 1500, 20, 1800.0, 900.0, 1.3, 1.0),  # 8 lanes
    (64, 640, 24, 700, 48, 900.0, 450.0, 1.1, 1.0),   # 8 lanes, several chunks
    (24, 24, 40, 90, 150, 90.0, 45.0, 0.4, 1.0),      # shadows of 4 columns and more rows
    (16, 16, 24, 200, 260, 60.0, 60.0, 0.18, 1.0),    # shadows wider than the slots
    (24, 24, 40, 40, 120, 20.0, 10.0, 0.9, 1.0),      # steep rays, corners near the source
    (24, 20, 30, 48, 60, 90.0, 45.0, 0.9, 0.7),       # slices that are not 1
    (70, 62, 61, 130, 110, 180.0, 90.0, 0.9, 1.0),    # over 2^18 voxels
]


@pytest.mark.parametrize("case", CASES, ids=[str(c[:5]) for c in CASES])
@pytest.mark.parametrize("angle", [0.0, 45.0, 90.0, 201.3])
def test_columns_equal_voxels(gpu, case, angle):
    import torch

    nx, ny, nz, na, nb, SO, OD, det, dz = case
    rng = np.random.default_rng(nx + nz)
    f = np.float32
    yd = ((np.arange(na) - na / 2.0 + 0.5) * det).astype(f)
    zd = ((np.arange(nb) - nb / 2.0 + 0.5) * det).astype(f)
    phi = f(np.deg2rad(angle))
    T = lambda a: torch.tensor(a, device=gpu)  # noqa: E731
    y, ydd, zdd = T(rng.standard_normal(na * nb).astype(f)), T(yd), T(zd)
    out = [torch.full((nx * ny * nz,), np.nan, device=gpu) for _ in range(4)]
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def call(x, sc):
        check(load().asdpocs_atx_device(
            P(x), P(y), P(sc), float(np.cos(phi)), float(np.sin(phi)), P(ydd), P(zdd), SO, OD, 0.7,
            det, det, dz, nx, ny, nz, na, nb,
            C.c_void_p(torch.cuda.current_stream().cuda_stream or None)))

    call(out[0], out[1])
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call(out[2], out[3])
    g.replay()
    torch.cuda.synchronize()
    h = [np.full(nx * ny * nz, np.nan, f) for _ in range(2)]
    pkg.Atx_cone_mf_gpu_new(h[0], y.cpu().numpy(), h[1], float(np.cos(phi)), float(np.sin(phi)),
                            yd, zd, SO, OD, 0.7, det, det, dz, nx, ny, nz, na, nb)
    out += [T(a) for a in h]
    for a, b in ((0, 2), (1, 3), (4, 2), (5, 3)):
        assert torch.equal(out[a].view(torch.int32), out[b].view(torch.int32))
    assert float(out[1].abs().max()) > 0


# A warp holds four (8 lanes) and two (16 lanes) voxel columns and the image
# reaches past the fan, so that columns without rays sit beside columns with
# some; nx, ny, nz, na, nb, SO, OD.
CUT = [(128, 128, 72, 257, 200, 541.0, 408.0), (160, 160, 48, 400, 120, 541.0, 408.0)]


def _fan(case):
    nx, na, SO, OD = case[0], case[3], case[5], case[6]
    return SO / (SO + OD) * na / nx  # voxel size at which the image fills the fan


@pytest.mark.parametrize("case", CUT, ids=[str(c[:5]) for c in CUT])
@pytest.mark.parametrize("angle", [27.0, 45.0, 135.0, 222.0, 315.0])
def test_columns_beside_the_fan(gpu, case, angle):
    """Host calls, whose workspace the call before left full of NaN, against
    the device call and the per-voxel form (captured)."""
    import torch

    nx, ny, nz, na, nb, SO, OD = case
    para = dict(SO=SO, OD=OD, vxlsize=_fan(case), nx=nx, ny=ny, nz=nz, na=na, nb=nb,
                phi=-angle / 180 * np.pi, detsize=1.0)
    y = np.random.default_rng(int(angle)).standard_normal(na * nb).astype(np.float32)
    pkg.imgTVGradMin3D(np.full((nx, ny, nz), np.nan), 0.1, 1, 0)
    x, sc = pkg.Atx_cone_gpu(y, para)
    f, vx = np.float32, _fan(case)
    T = lambda a: torch.tensor(np.asarray(a, f), device=gpu)  # noqa: E731
    import oracle
    g = oracle.gateway_geometry(para["phi"], SO, OD, vx, 1.0, na, nb)
    yt, yd, zd = T(y), T(g["y_det"]), T(g["z_det"])
    out = [torch.full((nx * ny * nz,), np.nan, device=gpu) for _ in range(4)]

    def call(a, b):
        check(load().asdpocs_atx_device(
            C.c_void_p(a.data_ptr()), C.c_void_p(yt.data_ptr()), C.c_void_p(b.data_ptr()),
            g["cos_phi"], g["sin_phi"], C.c_void_p(yd.data_ptr()), C.c_void_p(zd.data_ptr()),
            g["SO"], g["OD"], g["scale"], g["det"], g["det"], 1.0, nx, ny, nz, na, nb,
            C.c_void_p(torch.cuda.current_stream().cuda_stream or None)))

    call(out[0], out[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(out[2], out[3])
    graph.replay()
    torch.cuda.synchronize()
    want = [o.cpu().numpy() for o in out[2:]]
    assert np.isfinite(want[0]).all() and (want[1] == 0).any() and (want[1] > 0).any()
    for got in ((out[0].cpu().numpy(), out[1].cpu().numpy()), (x, sc)):
        for a, b in zip(got, want):
            assert np.array_equal(a.ravel(), b)


@pytest.mark.parametrize("case", CUT, ids=[str(c[:5]) for c in CUT])
def test_plan_of_columns_beside_the_fan(gpu, case, monkeypatch):
    """The same in a plan whose first view is at 0 degrees (odd bins: a ray
    along the axis, whose slopes are infinite): the per-voxel plan's image."""
    nx, ny, nz, na, nb, SO, OD = case
    phi = np.array([0.0, 27.0, 45.0, 135.0, 315.0])
    para = dict(SO=SO, OD=OD, vxlsize=_fan(case), nx=nx, ny=ny, nz=nz, na=na, nb=nb, detsize=1.0,
                phi_vec=phi, maxnumIter=2, numOfgradients=2, alpha=0.002)
    P = np.random.default_rng(nz).random(na * nb * len(phi)).astype(np.float32)

    def image():
        with pkg.Plan([para], [phi]) as pl:
            pl.set_sinogram(0, P)
            pl.reset()
            pl.run()
            return np.asarray(pl.image(0))

    got = image()
    monkeypatch.setenv("ASDPOCS_CONE_ATX", "voxel")
    want = image()
    assert np.isfinite(want).all() and np.array_equal(got, want)


# Sizes at which a plan's columns have 2, 4, 8 and 16 lanes, whole segments of
# slices that no ray crosses, chunks that begin inside a segment, and the walk's
# segments end early: nx, ny, nz, na, nb, part of the fan the image fills.
FEW = [(64, 90, 2, 110, 6, 1.0), (70, 90, 3, 131, 2, 1.3), (64, 160, 7, 150, 15, 1.0),
       (40, 160, 100, 161, 9, 1.2), (33, 95, 65, 100, 40, 1.0), (40, 100, 40, 80, 1, 1.0),
       (96, 70, 20, 96, 60, 2.0)]


@pytest.mark.parametrize("case", FEW, ids=[str(c[:5]) for c in FEW])
@pytest.mark.parametrize("bad", [False, True])
def test_forms_of_the_plan_step_agree(gpu, case, bad, monkeypatch):
    """A plan's backward step per voxel, in columns and walked, over volumes of
    which a view crosses few slices or few columns: the same bits, also with a
    sinogram value that is not finite (whole windows) and for two instances of
    different sizes in one launch."""
    nx, ny, nz, na, nb, fill = case
    phi = np.array([0.0, 33.0, 45.0, 118.0, 290.0])
    vx = 400.0 / 700.0 * na / max(nx, ny) * fill
    para = dict(SO=400.0, OD=300.0, vxlsize=vx, nx=nx, ny=ny, nz=nz, na=na, nb=nb, detsize=1.0,
                phi_vec=phi, maxnumIter=2, numOfgradients=2, alpha=0.002)
    ps = [para, dict(para, nx=nx - 9, nz=max(2, nz - 5), nb=nb + 2)]
    rng = np.random.default_rng(nx + nz)
    Ps = [rng.random(p["na"] * p["nb"] * len(phi)).astype(np.float32) for p in ps]
    if bad:
        Ps[0][na * nb + na // 2] = np.inf

    def images(form):
        monkeypatch.setenv("ASDPOCS_CONE_ATX", form)
        with pkg.Plan(ps, [phi] * 2) as pl:
            for k in range(2):
                pl.set_sinogram(k, Ps[k])
            pl.reset()
            pl.run()
            return [pl.image(k) for k in range(2)]

    want = images("voxel")
    assert bad or np.isfinite(want[0]).all()
    assert np.abs(want[1]).max() > 0
    for form in ("columns", "walk", ""):
        for a, b in zip(images(form), want):
            assert np.array_equal(a, b, equal_nan=True), form


@pytest.mark.parametrize("dims", [(256, 256, 4, 400, 7), (256, 256, 8, 400, 14),
                                  (256, 256, 24, 400, 13), (128, 128, 48, 220, 30)])
def test_device_step_beside_a_few_crossed_slices(gpu, oracle_mod, dims):
    """asdpocs_atx_device on both sides of its choice of form, against the form
    it takes under capture."""
    import torch

    nx, ny, nz, na, nb = dims
    f = np.float32
    g = oracle_mod.gateway_geometry(-0.7, 541.0, 408.0, 541.0 / 949.0 * na / nx, 1.0, na, nb)
    T = lambda a: torch.tensor(np.asarray(a, f), device=gpu)  # noqa: E731
    y = T(np.random.default_rng(nz).standard_normal(na * nb))
    yd, zd = T(g["y_det"]), T(g["z_det"])
    out = [torch.full((nx * ny * nz,), np.nan, device=gpu) for _ in range(4)]

    def call(x, sc):
        check(load().asdpocs_atx_device(
            C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), C.c_void_p(sc.data_ptr()),
            g["cos_phi"], g["sin_phi"], C.c_void_p(yd.data_ptr()), C.c_void_p(zd.data_ptr()),
            g["SO"], g["OD"], g["scale"], g["det"], g["det"], 1.0, nx, ny, nz, na, nb,
            C.c_void_p(torch.cuda.current_stream().cuda_stream or None)))

    call(out[0], out[1])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(out[2], out[3])
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])
    assert float(out[1].max()) > 0
