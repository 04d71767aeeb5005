"""Performance cases: the work users have this package do, through its public entry points.

A case is a dict of plain values; ``kind`` says which entry points it runs:

* ``mex_pair``     one view through the drop-in gateways ``Ax_cone_gpu`` and ``Atx_cone_gpu``
                   (host arrays in and out), as the reference's drivers call them in every step;
* ``device_pair``  a scan's views projected and back-projected between device buffers
                   (``asdpocs_ax_device``, ``asdpocs_atx_device``): a program with its own iteration;
* ``forward`` / ``back``  one direction of that, for volumes;
* ``tv_mex``       TV steepest descent of a double image in host memory
                   (``imgTVGradMin``, ``imgTVGradMin3D``);
* ``tv_device``    the same on a float image in device memory (``asdpocs_tv_device``);
* ``one_call``     a whole reconstruction by ``ASD_POCS_cuda``, plan creation included;
* ``plan``         device-resident reconstructions through ``Plan``: a scan's sinograms are set,
                   the plan runs, the images stay on the device.  ``batch`` instances of one
                   protocol, or (``mix``) of sizes and view counts spread over a range.

Scans and images are sums of random ellipses (ellipsoids); sinograms are their
line integrals in closed form with Poisson noise, so no input comes from the
code under test.  The reconstructions use the small TV step (alpha 0.002) at
which the iteration is well conditioned; the cost does not depend on it.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

import asd_pocs_mex_cuda_demo_gb300 as pkg

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call there is: one fan-beam view of a 64^2 image through both gateways
        dict(name="mex_pair_64", kind="mex_pair", nx=64, ny=64, nz=1, na=128, nb=1, nv=1),
        # a sparse-view head slice's 60 views, device buffers, both directions
        dict(name="device_pair_fan_512", kind="device_pair", nx=512, ny=512, nz=1, na=888, nb=1,
             nv=60),
        # a few views of a 256^3 cone-beam volume on a 512^2 detector, device buffers
        dict(name="forward_cone_256", kind="forward", nx=256, ny=256, nz=256, na=512, nb=512, nv=4,
             exact=False),
        dict(name="back_cone_256", kind="back", nx=256, ny=256, nz=256, na=512, nb=512, nv=4),
        # the TV functions by themselves, 20 steps as in the drivers
        dict(name="tv_mex_256", kind="tv_mex", nx=256, ny=256, nz=1, steps=20),
        dict(name="tv_mex_128x128x128", kind="tv_mex", nx=128, ny=128, nz=128, steps=20),
        dict(name="tv_device_256x256x256", kind="tv_device", nx=256, ny=256, nz=256, steps=20),
        # a small reconstruction in one call, as a MATLAB user's first run
        dict(name="one_call_fan_64", kind="one_call", nx=64, ny=64, nz=1, na=128, nb=1, nv=24,
             iters=5),
        # one head slice on the device
        dict(name="plan_fan_512", kind="plan", nx=512, ny=512, nz=1, na=888, nb=1, nv=60, batch=1,
             iters=10, storage="f32", exact=False, mix=0),
        # a batch of 64 slices of one protocol: the throughput workload
        dict(name="plan_fan_512_batch64", kind="plan", nx=512, ny=512, nz=1, na=888, nb=1, nv=60,
             batch=64, iters=4, storage="f32", exact=False, mix=0),
        # slices of several sizes and view counts in one plan, sinograms in FP16
        dict(name="plan_uneven", kind="plan", nx=512, ny=512, nz=1, na=768, nb=1, nv=120, batch=24,
             iters=2, storage="f16", exact=False, mix=7),
        # one cone-beam volume, 60 of its views
        dict(name="plan_cone_256", kind="plan", nx=256, ny=256, nz=256, na=512, nb=512, nv=60,
             batch=1, iters=1, storage="f32", exact=False, mix=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fan_sizes(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return dict(nx=n, ny=max(lo // 2, int(n * rng.choice((1, 1, 0.83)))), nz=1,
                na=int(n * rng.uniform(1.4, 2.0)), nb=1)


def _cone_sizes(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    return dict(nx=n, ny=int(n * rng.choice((1, 1, 0.9))), nz=int(n * rng.uniform(0.4, 1.0)),
                na=int(n * rng.uniform(1.4, 2.0)), nb=int(n * rng.uniform(1.0, 2.0)))


def draw(rng):
    kind = rng.choice(("mex_pair", "device_pair", "forward", "back", "tv_mex", "tv_device",
                       "one_call", "plan_fan", "plan_batch", "plan_uneven", "plan_cone"))
    if kind == "mex_pair":
        sizes = _fan_sizes(rng, 48, 768) if rng.random() < 0.5 else _cone_sizes(rng, 24, 128)
        return dict(kind=kind, nv=1, **sizes)
    if kind == "device_pair":
        return dict(kind=kind, nv=rng.randint(20, 120), **_fan_sizes(rng, 64, 768))
    if kind in ("forward", "back"):
        case = dict(kind=kind, nv=rng.randint(2, 6), **_cone_sizes(rng, 48, 256))
        if kind == "forward":
            case["exact"] = rng.random() < 0.3  # the exact (Siddon) lengths
        return case
    if kind in ("tv_mex", "tv_device"):
        if rng.random() < 0.5:
            nx, ny, nz = _log_int(rng, 48, 1024), _log_int(rng, 48, 1024), 1
        else:
            top = 128 if kind == "tv_mex" else 256
            nx, ny, nz = (_log_int(rng, 24, top) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.choice((1, 5, 20, 20)))
    if kind == "one_call":
        return dict(kind=kind, nv=rng.randint(12, 60), iters=rng.randint(2, 8),
                    **_fan_sizes(rng, 48, 256))
    more = dict(kind="plan", storage=rng.choice(("f32", "f32", "f16", "bf16")), exact=False, mix=0)
    if kind == "plan_fan":
        more["exact"] = rng.random() < 0.2
        return dict(batch=1, nv=rng.randint(24, 120), iters=rng.randint(2, 10), **more,
                    **_fan_sizes(rng, 64, 768))
    if kind == "plan_batch":
        return dict(batch=rng.randint(2, 64), nv=rng.randint(24, 60), iters=rng.randint(1, 3),
                    **more, **_fan_sizes(rng, 64, 512))
    if kind == "plan_uneven":
        more["mix"] = rng.randint(1, 999)
        return dict(batch=rng.randint(4, 24), nv=rng.randint(40, 120), iters=rng.randint(1, 2),
                    **more, **_fan_sizes(rng, 128, 512))
    more["exact"] = rng.random() < 0.2
    return dict(batch=rng.choice((1, 1, 3)), nv=rng.randint(8, 24), iters=rng.randint(1, 2), **more,
                **_cone_sizes(rng, 32, 160))


# ------------------------------------------------- geometry, phantoms and scans
def _geometry(c):
    """The para fields of a case: a fan-beam gantry, or a cone-beam one; the
    detector is as wide at every bin count and the image fills its view."""
    SO, OD, wide = (541.0, 408.0, 888.0) if c["nz"] == 1 else (1000.0, 500.0, 409.6)
    det = wide / c["na"]
    vxl = SO / (SO + OD) * wide / max(c["nx"], c["ny"])
    return dict(SO=SO, OD=OD, vxlsize=vxl, detsize=det, nx=c["nx"], ny=c["ny"], nz=c["nz"],
                na=c["na"], nb=c["nb"])


def _views(nv):
    return np.arange(1, nv + 1, dtype=np.float64) * (360.0 / nv)


def _launcher(g, phi_deg):
    """What the gateways pass on for one view (single precision, voxel units)."""
    f = np.float32
    phi = f(-phi_deg / 180.0 * math.pi)
    s = f(g["vxlsize"])
    det = f(f(g["detsize"]) / s)
    y = ((np.arange(g["na"]) - g["na"] / 2.0 + 0.5) * float(det)).astype(f)
    z = ((np.arange(g["nb"]) - g["nb"] / 2.0 + 0.5) * float(det)).astype(f)
    return dict(cos=f(np.cos(phi)), sin=f(np.sin(phi)), SO=f(f(g["SO"]) / s), OD=f(f(g["OD"]) / s),
                scale=s, det=det, y=y, z=z)


def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _ellipses(seed, planar, count=12):
    """Rows (amplitude /mm, centre, semi-axes, angle in the plane), lengths
    relative to the image's half width: a body and inserts in it."""
    r = random.Random(int(seed))
    rows = [(0.02, 0.0, 0.0, 0.0, r.uniform(0.7, 0.85), r.uniform(0.75, 0.9), 0.8, 0.0)]
    for _ in range(count):
        rows.append((r.choice((-0.009, -0.004, 0.003, 0.008)), r.uniform(-0.45, 0.45),
                     r.uniform(-0.45, 0.45), 0.0 if planar else r.uniform(-0.4, 0.4),
                     r.uniform(0.03, 0.25), r.uniform(0.03, 0.25), r.uniform(0.05, 0.25),
                     r.uniform(0.0, math.pi)))
    return rows


def _image(g, rows):
    """The ellipses on the voxel grid, [nz, ny, nx] double."""
    n = max(g["nx"], g["ny"])
    ax = [(torch.arange(k, device=DEV, dtype=F64) - k // 2 + 0.5) / (n / 2)
          for k in (g["nx"], g["ny"], g["nz"])]
    x, y, z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    if g["nz"] == 1:
        z = torch.zeros_like(z)
    out = torch.zeros(g["nz"], g["ny"], g["nx"], device=DEV, dtype=F64)
    for amp, x0, y0, z0, a, b, c, t in rows:
        u = (x - x0) * math.cos(t) + (y - y0) * math.sin(t)
        v = (y - y0) * math.cos(t) - (x - x0) * math.sin(t)
        out += amp * ((u / a) ** 2 + (v / b) ** 2 + ((z - z0) / c) ** 2 <= 1)
    return out.clamp_(min=0.0)


def _scan(g, phis, rows, seed):
    """Noisy sinogram [nv, nb*na] float: -ln of Poisson counts (1e5 per bin)
    behind the ellipses, their chords in closed form."""
    L = _launcher(g, 0.0)
    half = max(g["nx"], g["ny"]) / 2.0
    th = torch.tensor(-phis / 180.0 * math.pi, device=DEV, dtype=F64)[:, None, None]
    co, si = th.cos(), th.sin()
    yd = torch.tensor(L["y"], device=DEV, dtype=F64)[None, None, :]
    zd = torch.tensor(L["z"], device=DEV, dtype=F64)[None, :, None]
    p = [-co * float(L["SO"]) / half, -si * float(L["SO"]) / half]
    d = [(co * float(L["OD"] + L["SO"]) - si * yd) / half,
         (si * float(L["OD"] + L["SO"]) + co * yd) / half, zd / half]
    length = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt() * half * g["vxlsize"]
    out = torch.zeros(len(phis), g["nb"], g["na"], device=DEV, dtype=F64)
    for amp, x0, y0, z0, a, b, c, t in rows:
        ct, st = math.cos(t), math.sin(t)
        pu = ((p[0] - x0) * ct + (p[1] - y0) * st) / a
        pv = ((p[1] - y0) * ct - (p[0] - x0) * st) / b
        du, dv = (d[0] * ct + d[1] * st) / a, (d[1] * ct - d[0] * st) / b
        pw, dw = -z0 / c, d[2] / c
        qa = du ** 2 + dv ** 2 + dw ** 2
        qb = pu * du + pv * dv + pw * dw
        disc = qb ** 2 - qa * (pu ** 2 + pv ** 2 + pw ** 2 - 1)
        out += amp * length * 2 * disc.clamp(min=0).sqrt() / qa
    counts = torch.poisson(1e5 * torch.exp(-out.clamp(min=0)), generator=_rng(seed)).clamp_(min=1)
    return -torch.log(counts / 1e5).reshape(len(phis), -1).float()


def _noise(shape, seed, size):
    return size * torch.randn(shape, device=DEV, dtype=F64, generator=_rng(seed))


# --------------------------------------------------------------------- prepare
class _DeviceArray:
    """A float buffer of the library's, for torch.as_tensor."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr="<f4",
                                             version=3)


def _instances(c):
    """The sizes of a plan's instances: one protocol, or sizes and view counts
    from a few protocols of the range (seeded by ``mix``)."""
    if not c["mix"]:
        return [dict(c) for _ in range(c["batch"])]
    r = random.Random(c["mix"])
    kinds = []
    for k in range(5):
        f = (1.0, 0.75, 0.65, 0.5, 0.5)[k]
        kinds.append(dict(c, nx=int(c["nx"] * f), ny=int(c["ny"] * f), na=int(c["na"] * f),
                          nv=max(8, int(c["nv"] * r.uniform(0.4, 1.0)))))
    return [dict(r.choice(kinds)) for _ in range(c["batch"])]


def _device_calls(c, x, y):
    """Buffers and ready argument lists of a scan's device calls."""
    g = _geometry(c)
    N, M = c["nx"] * c["ny"] * c["nz"], c["na"] * c["nb"]
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    L0 = _launcher(g, 0.0)
    s = dict(kind=c["kind"], g=g, exact=c.get("exact", False), x=x, y=y,
             yd=torch.tensor(L0["y"], device=DEV), zd=torch.tensor(L0["z"], device=DEV),
             fwd=[], back=[])
    nv = c["nv"]
    s["out_y"], s["out_sr"] = (torch.empty(nv, M, device=DEV) for _ in range(2))
    s["out_x"], s["out_sc"] = (torch.empty(nv if y is not None else 0, N, device=DEV)
                               for _ in range(2))
    dims = [C.c_int(c[k]) for k in ("nx", "ny", "nz", "na", "nb")]
    for v, phi in enumerate(_views(nv)):
        L = _launcher(g, phi)
        ang = [C.c_float(float(L["cos"])), C.c_float(float(L["sin"])), P(s["yd"]), P(s["zd"]),
               C.c_float(float(L["SO"])), C.c_float(float(L["OD"])), C.c_float(float(L["scale"]))]
        det = C.c_float(float(L["det"]))
        if x is not None:
            s["fwd"].append([P(x), P(s["out_y"][v]), P(s["out_sr"][v]), *ang, C.c_float(1.0),
                             *dims])
        if y is not None:
            s["back"].append([P(s["out_x"][v]), P(y[v]), P(s["out_sc"][v]), *ang, det, det,
                              C.c_float(1.0), *dims])
    return s


def prepare(case, seed):
    c, kind = dict(case), case["kind"]
    g = _geometry(c) if "na" in c else None
    rows = _ellipses(seed, c["nz"] == 1)
    if kind == "mex_pair":
        phi = random.Random(seed + 1).uniform(0.0, 360.0)
        x = _image(g, rows).float().cpu().numpy().ravel()
        y = _scan(g, np.array([phi]), rows, seed)[0].cpu().numpy()
        return dict(kind=kind, x=x, y=y, para=dict(g, phi=-phi / 180.0 * math.pi))
    if kind in ("device_pair", "forward", "back"):
        x = y = None
        if kind != "back":
            im = _image(g, rows)
            x = (im + _noise(im.shape, seed + 1, 5e-4)).clamp_(min=0.0).float().reshape(-1)
        if kind != "forward":
            y = _scan(g, _views(c["nv"]), rows, seed) * 0.1 \
                + _noise((c["nv"], c["na"] * c["nb"]), seed + 2, 0.02).float()
        return _device_calls(c, x, y)
    if kind in ("tv_mex", "tv_device"):
        im = _image(dict(nx=c["nx"], ny=c["ny"], nz=c["nz"]), rows)
        old = im + _noise(im.shape, seed + 1, 1e-3)
        im = im + _noise(im.shape, seed + 2, 2e-3)
        s = dict(kind=kind, steps=c["steps"], dims=(c["nx"], c["ny"], c["nz"]))
        if kind == "tv_device":
            return dict(s, im=im.float().contiguous(), old=old.float().contiguous())
        # column-major (MATLAB) arrays
        shape = s["dims"] if c["nz"] > 1 else s["dims"][:2]
        F = lambda t: t.cpu().numpy().ravel().reshape(shape, order="F")  # noqa: E731
        return dict(s, im=F(im), old=F(old))
    if kind == "one_call":
        phis = _views(c["nv"])
        P = _scan(g, phis, rows, seed).double().cpu().numpy()
        return dict(kind=kind, P=P.T, para=dict(g, phi_vec=phis, maxnumIter=c["iters"],
                                                alpha=0.002))
    insts = _instances(c)
    paras, phis, scans = [], [], []
    for k, i in enumerate(insts):
        gi = _geometry(i)
        paras.append(dict(gi, maxnumIter=c["iters"], alpha=0.002, sino_storage=c["storage"],
                          ax_mode="exact" if c["exact"] else "reference"))
        phis.append(_views(i["nv"]))
        scans.append(_scan(gi, phis[-1], _ellipses(1000 * seed + k, c["nz"] == 1),
                           1000 * seed + k).contiguous())
    torch.cuda.synchronize()
    plan = pkg.Plan(paras, phis)
    images = [torch.as_tensor(_DeviceArray(plan.image_ptr(k), (plan.voxels(k),)), device=DEV)
              for k in range(len(insts))]
    return dict(kind=kind, plan=plan, scans=scans, images=images)


# ------------------------------------------------------------------------- run
def _ok(rc):
    if rc:
        raise RuntimeError(pkg.load().asdpocs_last_error().decode())


def run(s):
    kind = s["kind"]
    if kind == "mex_pair":
        y, sr = pkg.Ax_cone_gpu(s["x"], s["para"])
        x, sc = pkg.Atx_cone_gpu(s["y"], s["para"])
        return dict(y=y, sr=sr, x=x, sc=sc)
    if kind in ("device_pair", "forward", "back"):
        lib, out = pkg.load(), {}
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream or None)
        ax = lib.asdpocs_ax_siddon_device if s["exact"] else lib.asdpocs_ax_device
        for k in range(max(len(s["fwd"]), len(s["back"]))):
            if s["fwd"]:
                _ok(ax(*s["fwd"][k], st))
            if s["back"]:
                _ok(lib.asdpocs_atx_device(*s["back"][k], st))
        if s["fwd"]:
            out.update(y=s["out_y"], sr=s["out_sr"])
        if s["back"]:
            out.update(x=s["out_x"], sc=s["out_sc"])
        return out
    if kind == "tv_mex":
        fn = pkg.imgTVGradMin3D if s["dims"][2] > 1 else pkg.imgTVGradMin
        return fn(s["im"], 0.02, s["steps"], 1, s["old"])
    if kind == "tv_device":
        im = s["im"].clone()
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream or None)
        _ok(pkg.load().asdpocs_tv_device(C.c_void_p(im.data_ptr()), C.c_void_p(s["old"].data_ptr()),
                                         *s["dims"], 0.02, s["steps"], 1, st))
        return im
    if kind == "one_call":
        m, out = pkg.ASD_POCS_cuda(s["P"], s["para"])
        # the driver widens its single-precision image to MATLAB's double
        return dict(m=m.astype(np.float32), dd=float(out["dataTolerance"]),
                    n=int(out["IterationNum"]))
    plan = s["plan"]
    for k, P in enumerate(s["scans"]):
        plan.set_sinogram(k, P.data_ptr())
    plan.reset()
    plan.run()
    # copies: the plan's own buffers go with the plan
    if len(s["images"]) > 1:
        return torch.cat(s["images"])
    st = plan.stats(0)
    return dict(m=s["images"][0].clone(), dd=float(st["dataTolerance"]), n=int(st["IterationNum"]))


# ------------------------------------------------------------------------ work
def work(case):
    """Inputs read once and outputs written once; two flops per ray-voxel
    crossing of a projection, about 20 per voxel of a TV step."""
    c, kind = case, case["kind"]
    N = c["nx"] * c["ny"] * c["nz"]
    if kind in ("tv_mex", "tv_device"):
        b = 8 if kind == "tv_mex" else 4
        return dict(bytes=3 * b * N, flops=20.0 * c["steps"] * N * (1 if c["nz"] == 1 else 1.5))

    def crossings(i):
        return i["na"] * i["nb"] * max(i["nx"], i["ny"]) * (1.25 if i["nz"] == 1 else 1.5)

    M, X = c["na"] * c["nb"], crossings(c)
    if kind == "mex_pair":
        return dict(bytes=12 * (N + M), flops=8.0 * X)
    if kind == "device_pair":
        return dict(bytes=4 * N + c["nv"] * (12 * M + 8 * N), flops=8.0 * X * c["nv"])
    if kind == "forward":
        return dict(bytes=4 * N + 8 * M * c["nv"], flops=4.0 * X * c["nv"])
    if kind == "back":
        return dict(bytes=8 * N * c["nv"] + 4 * M * c["nv"], flops=4.0 * X * c["nv"])
    total = dict(bytes=0.0, flops=0.0)
    for i in [c] if kind == "one_call" else _instances(c):
        Ni = i["nx"] * i["ny"] * i["nz"]
        size = 8 if kind == "one_call" else 4 if c["storage"] == "f32" else 2
        total["bytes"] += size * i["nv"] * i["na"] * i["nb"] + (8 if kind == "one_call" else 4) * Ni
        total["flops"] += c["iters"] * (8.0 * crossings(i) * i["nv"]
                                        + 20 * 20.0 * Ni * (1 if i["nz"] == 1 else 1.5))
    return total


# ----------------------------------------------- the same results in 64 bits
def _march(vol, g, L):
    """The forward projector of Ax_cone_gpu in double: each ray's columns along
    its driving axis, split where it crosses a row or a slice."""
    nx, ny, nz = g["nx"], g["ny"], g["nz"]
    c, s, SO, OD = (float(L[k]) for k in ("cos", "sin", "SO", "OD"))
    yd = torch.tensor(L["y"], device=DEV, dtype=F64)
    zd = torch.tensor(L["z"], device=DEV, dtype=F64)
    yd, zd = yd.repeat(g["nb"]), zd.repeat_interleave(g["na"])
    x1, y1 = -c * SO, -s * SO
    x2, y2 = c * OD - s * yd, s * OD + c * yd
    y = torch.zeros(yd.numel(), device=DEV, dtype=F64)
    sr = torch.zeros_like(y)
    flat = vol.reshape(-1)
    xdrive = (x1 - x2).abs() > (y1 - y2).abs()
    for xd in (True, False):
        rays = torch.nonzero(xdrive == xd).reshape(-1)
        nu, nv, su, sv = (nx, ny, 1, nx) if xd else (ny, nx, nx, 1)
        us, vs = (x1, y1) if xd else (y1, x1)
        ue = torch.arange(nu + 1, device=DEV, dtype=F64) - nu // 2
        iu = torch.arange(nu, device=DEV)
        for r in rays.split(max(1, 6_000_000 // nu)):
            du = ((x2 - x1) if xd else (y2 - y1))[r, None]
            dv = ((y2 - y1) if xd else (x2 - x1))[r, None]
            ve = vs + dv / du * (ue - us) + nv // 2
            we = zd[r, None] / du * (ue - us) + nz // 2
            v1, v2 = torch.minimum(ve[:, :-1], ve[:, 1:]), torch.maximum(ve[:, :-1], ve[:, 1:])
            w1, w2 = torch.minimum(we[:, :-1], we[:, 1:]), torch.maximum(we[:, :-1], we[:, 1:])

            def split(a1, a2, n):
                i1, i2 = a1.floor().long(), a2.floor().long()
                cut = i1 != i2
                mid = (i2 > 0) & (i2 < n)
                lo = torch.where(cut, mid | (i2 == n), torch.ones_like(cut)) & (i1 >= 0) & (i1 < n)
                hi = cut & (mid | (i2 == 0)) & (i2 >= 0) & (i2 < n)
                frac = torch.where(cut, (i2 - a1) / (a2 - a1).clamp(min=1e-300),
                                   torch.ones_like(a1))
                return i1, i2, lo, hi, frac

            iv1, iv2, vlo, vhi, rv = split(v1, v2, nv)
            iw1, iw2, wlo, whi, rw = split(w1, w2, nz)
            l = (((v2 - v1) ** 2 + 1) * (1 + zd[r, None] ** 2 / (du ** 2 + dv ** 2))).sqrt()
            vf = rv <= rw
            pieces = ((torch.minimum(rv, rw), iv1, iw1, vlo & wlo),
                      ((rv - rw).abs(), torch.where(vf, iv2, iv1), torch.where(vf, iw1, iw2),
                       torch.where(vf, vhi & wlo, vlo & whi)),
                      (1 - torch.maximum(rv, rw), iv2, iw2, vhi & whi))
            for frac, iv, iw, on in pieces:
                w = torch.where(on, frac * l, torch.zeros_like(l))
                at = iu * su + iv.clamp(0, nv - 1) * sv + iw.clamp(0, nz - 1) * (nx * ny)
                y[r] += (w * flat[at]).sum(1)
                sr[r] += w.sum(1)
    return y, sr


def _pairs(g, L, vox):
    """Bins and chords of the voxels ``vox`` (flat indices): ([n, K] ray
    indices, [n, K] lengths in voxel widths, 0 where a ray passes by)."""
    nx, ny, nz, na, nb = (g[k] for k in ("nx", "ny", "nz", "na", "nb"))
    c, s, SO, OD, det = (float(L[k]) for k in ("cos", "sin", "SO", "OD", "det"))
    x = (vox % nx - nx // 2).double() + 0.5
    y = (vox // nx % ny - ny // 2).double() + 0.5
    z = (vox // (nx * ny) - nz // 2).double() + 0.5
    xr, yr = c * x + s * y, c * y - s * x
    t = (SO + OD) / ((xr + SO) * det)
    a0, b0 = ((yr - 1) * t + na // 2).floor().long(), ((z - 1) * t + nb // 2).floor().long()
    ka = int((((yr + 1) * t + na // 2).floor().long() - a0).max()) + 1
    kb = int((((z + 1) * t + nb // 2).floor().long() - b0).max()) + 1 if nb > 1 or nz > 1 else 1
    if kb == 1:
        b0 = torch.zeros_like(b0)
    ia = (a0[:, None, None] + torch.arange(ka, device=DEV)).expand(-1, kb, -1)
    ib = (b0[:, None, None] + torch.arange(kb, device=DEV)[:, None]).expand(-1, -1, ka)
    ok = (ia >= 0) & (ia < na) & (ib >= 0) & (ib < nb)
    ia, ib = ia.clamp(0, na - 1), ib.clamp(0, nb - 1)
    yd = torch.tensor(L["y"], device=DEV, dtype=F64)[ia]
    zd = torch.tensor(L["z"], device=DEV, dtype=F64)[ib]
    p = [-c * SO - x, -s * SO - y, -z]
    d = [c * OD - s * yd + c * SO, s * OD + c * yd + s * SO, zd]
    if nz == 1 and nb == 1:
        p, d = p[:2], d[:2]
    lo = torch.full_like(yd, -math.inf)
    hi = torch.full_like(yd, math.inf)
    for pk, dk in zip(p, d):
        pk = pk[:, None, None].expand_as(yd)
        still = dk == 0
        e = torch.where(still, torch.ones_like(dk), dk)
        u, v = (-0.5 - pk) / e, (0.5 - pk) / e
        inside = still & (pk.abs() <= 0.5)
        far = torch.full_like(u, math.inf)
        lo = torch.maximum(lo, torch.where(still, torch.where(inside, -far, far),
                                           torch.minimum(u, v)))
        hi = torch.minimum(hi, torch.where(still, torch.where(inside, far, -far),
                                           torch.maximum(u, v)))
    length = sum(dk * dk for dk in d).sqrt() * (hi - lo).clamp(min=0)
    length = torch.where(ok, length, torch.zeros_like(length))
    return (ib * na + ia).reshape(len(vox), -1), length.reshape(len(vox), -1)


def _back(g, L, y):
    """Back-projection and column sums of one view, without the scale."""
    N = g["nx"] * g["ny"] * g["nz"]
    x, sc = (torch.empty(N, device=DEV, dtype=F64) for _ in range(2))
    for vox in torch.arange(N, device=DEV).split(1_000_000):
        idx, l = _pairs(g, L, vox)
        x[vox], sc[vox] = (l * y[idx]).sum(1), l.sum(1)
    return x, sc


def _tv(u, alpha, old, steps):
    """Steps of the TV descent on [B, nz, ny, nx] doubles, then positivity."""
    is3d = u.shape[1] > 1
    norm = lambda t: t.reshape(t.shape[0], -1).norm(dim=1).reshape(-1, 1, 1, 1)  # noqa: E731
    dist = norm(u - old)
    for _ in range(steps):
        p = torch.nn.functional.pad(u, (1, 1, 1, 1, 1, 1) if is3d else (1, 1, 1, 1))

        def at(dx=0, dy=0, dz=0):
            q = p[:, 1 + dz:p.shape[1] - 1 + dz] if is3d else p
            return q[:, :, 1 + dy:q.shape[2] - 1 + dy, 1 + dx:q.shape[3] - 1 + dx]

        f, xp, yp = at(), at(1), at(0, 1)
        sq = lambda *t: (1e-8 + sum(k * k for k in t)).sqrt()  # noqa: E731
        if is3d:
            zp = at(0, 0, 1)
            v = (6 * f - 2 * (at(-1) + at(0, -1) + at(0, 0, -1))) \
                / sq(f - at(-1), f - at(0, -1), f - at(0, 0, -1))
            v = v + 2 * (f - zp) / sq(zp - at(-1, 0, 1), zp - at(0, -1, 1), zp - f)
            v = v + 2 * (f - yp) / sq(yp - at(-1, 1), yp - f, yp - at(0, 1, -1))
            v = v + 2 * (f - xp) / sq(xp - f, xp - at(1, -1), xp - at(1, 0, -1))
        else:
            v = (2 * f - at(-1) - at(0, -1)) / sq(f - at(-1), f - at(0, -1))
            v = v - (xp - f) / sq(xp - f, xp - at(1, -1)) - (yp - f) / sq(yp - f, yp - at(-1, 1))
        u = u - alpha * dist / norm(v) * v
    return u.clamp(min=0.0)


def _reconstruct(g, phis, P, iters):
    """ASD-POCS of a batch of scans P [B, nv, M] of one geometry in double:
    (images [B, N], squared data residual of the last sweep [B], sweeps)."""
    N, B = g["nx"] * g["ny"] * g["nz"], P.shape[0]
    scale, planar = float(np.float32(g["vxlsize"])), g["nz"] == 1 and g["nb"] == 1
    Ls = [_launcher(g, p) for p in phis]
    tabs = [_pairs(g, L, torch.arange(N, device=DEV)) for L in Ls] if planar else None
    m = torch.zeros(N, B, device=DEV, dtype=F64)
    pre, first = m.clone(), m.clone()
    alpha, beta = torch.full((B,), 0.002, device=DEV, dtype=F64), 1.0
    grid = lambda t: t.T.reshape(B, g["nz"], g["ny"], g["nx"])  # noqa: E731
    for _ in range(iters):
        dd = torch.zeros(B, device=DEV, dtype=F64)
        for v, L in enumerate(Ls):
            if planar:
                idx, l = tabs[v]
                y = torch.zeros(g["na"], B, device=DEV, dtype=F64)
                y.index_add_(0, idx.reshape(-1), (l[:, :, None] * m[:, None, :]).reshape(-1, B))
                sr = torch.zeros(g["na"], device=DEV, dtype=F64)
                sr.index_add_(0, idx.reshape(-1), l.reshape(-1))
            else:
                y, sr = (t[:, None] for t in _march(m[:, 0], g, L))
                sr = sr[:, 0]
            sr = torch.where(sr == 0, torch.ones_like(sr), sr * scale)
            res = P[:, v].T - y * scale
            dd += (res * res).sum(0)
            cor = res / sr[:, None]
            if planar:
                bp, sc = (l[:, :, None] * cor[idx]).sum(1), l.sum(1)
            else:
                bp, sc = _back(g, L, cor[:, 0])
                bp = bp[:, None]
            sc = torch.where(sc == 0, torch.ones_like(sc), sc)
            m = (m + beta * bp / sc[:, None]).clamp(min=0.0)
        res_m, dp = m, (m - pre).norm(dim=0)
        m = _tv(grid(m), alpha.reshape(-1, 1, 1, 1), grid(first), 20).reshape(B, N).T
        dg = (m - res_m).norm(dim=0)
        alpha = torch.where(dg > 0.95 * dp, alpha * 0.95, alpha)
        beta, pre = beta * 0.995, m
    return res_m.T, dd, iters


def _stored(P, storage):
    return {"f16": P.half(), "bf16": P.bfloat16()}.get(storage, P).double()


def exact(case, seed):
    c, kind = case, case["kind"]
    if c.get("exact") or (kind == "plan" and c["nz"] > 1
                          and c["nv"] * c["iters"] * c["nx"] * c["ny"] * c["nz"] > 3e8):
        return None  # Siddon lengths and long volume scans are left to the bound of their type
    if kind == "plan":
        insts = _instances(c)
        out, dd = [None] * len(insts), 0.0
        groups = {}
        for k, i in enumerate(insts):
            groups.setdefault((i["nx"], i["ny"], i["nv"]) if c["nz"] == 1 else k, []).append(k)
        for ks in groups.values():
            i = insts[ks[0]]
            g, phis = _geometry(i), _views(i["nv"])
            P = torch.stack([_stored(_scan(g, phis, _ellipses(1000 * seed + k, c["nz"] == 1),
                                           1000 * seed + k), c["storage"]) for k in ks])
            m, dd, n = _reconstruct(g, phis, P, c["iters"])
            for k, im in zip(ks, m):
                out[k] = im
        if len(insts) > 1:
            return torch.cat(out)
        return dict(m=out[0], dd=float(dd[0]), n=n)
    s = prepare(case, seed)
    if kind == "one_call":
        g = _geometry(c)
        P = torch.tensor(s["P"].T.copy(), device=DEV)[None]
        m, dd, n = _reconstruct(g, _views(c["nv"]), P, c["iters"])
        shape = (c["nx"], c["ny"], c["nz"])
        return dict(m=m[0].cpu().numpy().reshape(shape, order="F"), dd=float(dd[0]), n=n)
    if kind in ("tv_mex", "tv_device"):
        nx, ny, nz = s["dims"]
        if kind == "tv_device":
            return _tv(s["im"].double()[None], 0.02, s["old"].double()[None], s["steps"])[0]
        T = lambda a: torch.tensor(a.ravel(order="F"), device=DEV).reshape(1, nz, ny, nx)  # noqa: E731
        r = _tv(T(s["im"]), 0.02, T(s["old"]), s["steps"]).cpu().numpy().ravel()
        return r.reshape(s["im"].shape, order="F")
    g = _geometry(c)
    scale = float(np.float32(g["vxlsize"]))
    if kind == "mex_pair":
        L = _launcher(g, -s["para"]["phi"] * 180.0 / math.pi)
        y, sr = _march(torch.tensor(s["x"], device=DEV).double(), g, L)
        x, sc = _back(g, L, torch.tensor(s["y"], device=DEV).double())
        return dict(y=y * scale, sr=sr * scale, x=x * scale, sc=sc * scale)
    out = {}
    Ls = [_launcher(g, p) for p in _views(c["nv"])]
    if kind != "back":
        r = [_march(s["x"].double(), g, L) for L in Ls]
        out.update(y=torch.stack([a for a, _ in r]) * scale,
                   sr=torch.stack([b for _, b in r]) * scale)
    if kind != "forward":
        r = [_back(g, L, y.double()) for L, y in zip(Ls, s["y"])]
        out.update(x=torch.stack([a for a, _ in r]) * scale,
                   sc=torch.stack([b for _, b in r]) * scale)
    return out
