"""GPU TV minimisation against the reference's src/tvmin results (golden
vectors) and the oracle.  FP64 entry points: relative L2 <= 1e-12; FP32
device variant: <= 1e-5."""
import numpy as np
import pytest

import asd_pocs_mex_cuda_demo_gb300 as pkg
from conftest import golden, rel_l2

pytestmark = pytest.mark.gpu


def test_tv_fp64_vs_reference_vectors(gpu):
    d = golden("tv.npz")
    assert rel_l2(pkg.imgTVGradMin(d["img2"], 0.2, 20, 1, d["old2"]), d["out2"]) < 1e-12
    assert rel_l2(pkg.imgTVGradMin(d["img2"] - 0.5, 0.05, 7, 0), d["out2_nopos"]) < 1e-12
    assert rel_l2(pkg.imgTVGradMin3D(d["img3"], 0.2, 20, 1, d["old3"]), d["out3"]) < 1e-12


@pytest.mark.parametrize("shape", [(1, 1), (5, 3), (64, 48), (257, 130)])
def test_tv2d_fp64_vs_oracle(gpu, oracle_mod, shape):
    rng = np.random.default_rng(shape[0])
    img = rng.random(shape)
    old = rng.random(shape)
    out = pkg.imgTVGradMin(img, 0.1, 5, 1, old)
    assert rel_l2(out, oracle_mod.tv(img, 0.1, 5, 1, old)) < 1e-12


@pytest.mark.parametrize("shape", [(3, 4, 2), (33, 20, 9), (64, 64, 32)])
def test_tv3d_fp64_vs_oracle(gpu, oracle_mod, shape):
    rng = np.random.default_rng(shape[2])
    img = rng.random(shape)
    out = pkg.imgTVGradMin3D(img, 0.05, 4, 1)
    assert rel_l2(out, oracle_mod.tv(img, 0.05, 4, 1)) < 1e-12


def test_tv_zero_iterations_and_constant_image(gpu, oracle_mod):
    img = np.random.default_rng(2).random((8, 8)) - 0.5
    out = pkg.imgTVGradMin(img, 0.2, 0, 1)
    assert np.array_equal(out, img)  # nTVIter == 0: no step and no clamp
    z = np.zeros((6, 6))
    o = pkg.imgTVGradMin(z, 0.2, 3, 0)
    r = oracle_mod.tv(z, 0.2, 3, 0)
    # the reference divides by a zero norm: 0/0 = NaN everywhere
    assert np.isnan(o).all() and np.isnan(r).all()


@pytest.mark.parametrize("shape", [(64, 48, 1), (128, 128, 1), (40, 36, 20)])
def test_tv_fp32_device_vs_oracle(gpu, oracle_mod, shape):
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    nx, ny, nz = shape
    rng = np.random.default_rng(nx + nz)
    img = rng.random(shape)
    old = rng.random(shape)
    t = torch.tensor(img.ravel(order="F"), dtype=torch.float32, device=gpu)
    o = torch.tensor(old.ravel(order="F"), dtype=torch.float32, device=gpu)
    s = torch.cuda.current_stream().cuda_stream
    check(load().asdpocs_tv_device(t.data_ptr(), o.data_ptr(), nx, ny, nz, 0.2, 10, 1, s))
    torch.cuda.synchronize()
    img32 = img.astype(np.float32).astype(np.float64)
    old32 = old.astype(np.float32).astype(np.float64)
    if nz == 1:
        img32, old32 = img32[:, :, 0], old32[:, :, 0]
    ref = oracle_mod.tv(img32, 0.2, 10, 1, old32)
    assert rel_l2(t.cpu().numpy(), ref.ravel(order="F")) < 1e-5


@pytest.mark.parametrize("steps", [1, 2, 5])
@pytest.mark.parametrize("shape", [(32, 16, 1), (33, 17, 1), (1, 40, 1), (31, 15, 1), (700, 9, 1),
                                   (32, 16, 2), (33, 17, 5), (7, 3, 67), (65, 48, 12)])
def test_tv_steps_at_tile_edges(gpu, oracle_mod, shape, steps):
    """Images that end at, before and after a tile of 32 x 16 and a slab of
    slices, in FP64 and FP32, with and without an old image."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    nx, ny, nz = shape
    rng = np.random.default_rng(nx * 31 + ny + nz)
    dims = shape if nz > 1 else shape[:2]
    img, old = rng.random(dims), rng.random(dims)
    fn = pkg.imgTVGradMin3D if nz > 1 else pkg.imgTVGradMin
    assert rel_l2(fn(img, 0.1, steps, 1, old), oracle_mod.tv(img, 0.1, steps, 1, old)) < 1e-12
    assert rel_l2(fn(img, 0.1, steps, 0), oracle_mod.tv(img, 0.1, steps, 0)) < 1e-12
    t, o = (torch.tensor(a.ravel(order="F"), dtype=torch.float32, device=gpu) for a in (img, old))
    f64 = [a.cpu().numpy().astype(np.float64).reshape(dims, order="F") for a in (t, o)]
    check(load().asdpocs_tv_device(t.data_ptr(), o.data_ptr(), nx, ny, nz, 0.1, steps, 1,
                                   torch.cuda.current_stream().cuda_stream))
    ref = oracle_mod.tv(f64[0], 0.1, steps, 1, f64[1])
    assert rel_l2(t.cpu().numpy(), ref.ravel(order="F")) < 1e-5


def test_tv_noalloc_large_image(gpu):
    """An image too large for three work images in the fixed scratch."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    a = torch.rand(1000 * 1001, device=gpu)
    b, old = a.clone(), torch.rand(1000 * 1001, device=gpu)
    s = torch.cuda.current_stream().cuda_stream
    check(load().asdpocs_tv_device(a.data_ptr(), old.data_ptr(), 1000, 1001, 1, 0.1, 4, 1, s))
    check(load().asdpocs_tv_device_noalloc(b.data_ptr(), old.data_ptr(), 1000, 1001, 1, 0.1, 4, 1,
                                           s))
    assert rel_l2(b.cpu().numpy(), a.cpu().numpy()) < 1e-5


@pytest.mark.parametrize("level", [1.4130100011825562, 1.4100697040557861, 1.0])
def test_tv_fp32_step_length_of_a_long_slab(gpu, level):
    """One FP32 step moves the image by alpha ||m - old||, whatever the stencil,
    so the length shows the two sums behind the step size.  The image is constant
    (equal squares, whose roundings add up instead of cancelling) and a slab has
    64 slices.  Bound, in units of 2^-24: a thread's four rows and their squares
    are rounded four times in each sum and the root halves that, 4; the step size,
    the product and the difference 3; 7 x 6e-8 = 4.2e-7."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    nx, ny, nz, alpha = 640, 960, 64, 10.0
    m = torch.full((nx * ny * nz,), level, dtype=torch.float32, device=gpu)
    old = torch.zeros_like(m)
    want = alpha * float(torch.linalg.vector_norm(m.double()))
    out = m.clone()
    check(load().asdpocs_tv_device(out.data_ptr(), old.data_ptr(), nx, ny, nz, alpha, 1, 0,
                                   torch.cuda.current_stream().cuda_stream))
    got = float(torch.linalg.vector_norm(out.double() - m.double()))
    assert abs(got / want - 1) < 4.2e-7, got / want - 1


def test_tv_fp32_infinite_distance(gpu):
    """A distance whose square overflows FP32 gives an infinite step, not NaN:
    voxels with a positive derivative go to -inf and positivity makes them 0."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    for dims in ((40, 33, 1), (40, 33, 9)):
        n = dims[0] * dims[1] * dims[2]
        m = torch.rand(n, device=gpu, generator=torch.Generator(gpu).manual_seed(1))
        old = torch.full_like(m, -3e19)
        check(load().asdpocs_tv_device(m.data_ptr(), old.data_ptr(), *dims, 0.1, 1, 1,
                                       torch.cuda.current_stream().cuda_stream))
        assert bool((torch.isinf(m) | (m == 0)).all())


@pytest.mark.parametrize("shape", [(31, 33, 24), (64, 64, 60), (40, 40, 301), (64, 64, 200)])
def test_tv3d_fp64_slab_lengths(gpu, oracle_mod, shape):
    """FP64 volumes whose items have one, two, eight and six slices."""
    rng = np.random.default_rng(shape[2])
    img, old = rng.random(shape), rng.random(shape)
    out = pkg.imgTVGradMin3D(img, 0.1, 3, 1, old)
    assert rel_l2(out, oracle_mod.tv(img, 0.1, 3, 1, old)) < 1e-12


def test_tv_device_with_room_for_one_work_image(gpu):
    """A volume whose three work images do not fit what is left of the device's
    memory: one is enough, as the result of a call with room shows.  An image of
    1 GiB and 2.2 GiB left."""
    import torch

    from asd_pocs_mex_cuda_demo_gb300._lib import check, load

    dims, n = (1024, 1024, 256), 1 << 28
    g = torch.Generator(gpu).manual_seed(5)
    a = torch.rand(n, device=gpu, generator=g)
    b = a.clone()
    st = torch.cuda.current_stream().cuda_stream
    torch.cuda.empty_cache()
    # the workspace gives up what it has first, so leave room for that, too
    left = (22 << 30) // 10
    hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device=gpu)
    try:
        check(load().asdpocs_tv_device(b.data_ptr(), None, *dims, 0.1, 3, 1, st))
    finally:
        del hold
        torch.cuda.empty_cache()
    check(load().asdpocs_tv_device(a.data_ptr(), None, *dims, 0.1, 3, 1, st))
    a, b = a.double(), b.double()
    assert float((a - b).norm() / a.norm()) < 1e-5
