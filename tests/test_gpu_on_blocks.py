"""Iterations on the caller's blocks (statistics asked for) beside the library's tiles (none): block
sizes, boundaries and block kernels at the benchmark's size and on small volumes, and the tile forms that need
large volumes.  Tolerance: 1e-5 relative L2 against the oracle and between runs on different blocks, 1e-6 an
iteration between tiles and blocks (float rounding of two transforms)."""
import os

import numpy as np
import pytest

import mvrgb300 as M
import oracle as O
import synthetic

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def rel(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.fixture(scope="module")
def data():
    ds = synthetic.config_256()
    return ds, [torch.from_numpy(a).cuda() for a in ds.images], [torch.from_numpy(a).cuda() for a in ds.weights]


@pytest.fixture(scope="module")
def plane_blocks(data):
    return run_256(data, (192, 192, 192), True)


def run_256(data, block, blocks, boundary=M.BOUNDARY_CIRCULAR):
    ds, imgs, ws = data
    with M.Deconvolution((256, 256, 256), 4, block, psf_type=M.PSF_OPTIMIZATION_I, lam=0.006, boundary=boundary,
                         weight_norm=M.WEIGHTS_HARD) as d:
        for v in range(4):
            d.set_view_device(v, imgs[v].data_ptr(), ws[v].data_ptr(), ds.psfs[v])
        d.prepare()
        d.run_iterations(2, stats=blocks)
        return d.get_psi()


@pytest.mark.parametrize("block,boundary", [
    ((192, 192, 192), M.BOUNDARY_REFERENCE),   # padded domains, mirror and value-1 extensions
    ((320, 320, 378), M.BOUNDARY_CIRCULAR),    # one block around the volume, row / column kernels
    ((256, 256, 256), M.BOUNDARY_CIRCULAR),    # pair or row / column kernels, 256-long columns
])
def test_full_size_block_grids(data, plane_blocks, block, boundary):
    assert rel(run_256(data, block, True, boundary), plane_blocks) <= 1e-5


def test_full_size_tiles_against_blocks(data, plane_blocks):
    assert rel(run_256(data, (192, 192, 192), False), plane_blocks) <= 2e-6


def volume(dims, kd, nv, seed):
    rng = np.random.default_rng(seed)
    shape = dims[::-1]
    imgs = [rng.uniform(5, 200, shape).astype(np.float32) for _ in range(nv)]
    ws = [rng.uniform(0.2, 0.9, shape).astype(np.float32) for _ in range(nv)]
    return imgs, ws, [synthetic.make_psf(kd, 1.0, 1.5, 40.0 * v) for v in range(nv)], rng.uniform(5, 150, shape).astype(np.float32)


def run(dims, block, mul, blocks, vol, its=1, boundary=M.BOUNDARY_REFERENCE):
    imgs, ws, psfs, psi = vol
    with M.Deconvolution(dims, len(imgs), block, mul=mul, psf_type=M.PSF_INDEPENDENT, lam=0.006, boundary=boundary) as d:
        for v in range(len(imgs)):
            d.set_view(v, imgs[v], ws[v], psfs[v])
        d.prepare()
        d.set_psi(psi)
        ks = [d.kernels(v, psfs[v].shape) for v in range(len(imgs))]
        mx = d.max_intensities()
        d.run_iterations(its, stats=blocks)
        return d.get_psi(), [k[0] for k in ks], [k[1] for k in ks], mx


@pytest.mark.parametrize("mul", [False, True])
def test_circular_blocks_of_a_small_volume(mul):
    dims, kd, block = (53, 41, 37), (5, 7, 5), (28, 32, 28)
    vol = volume(dims, kd, 2, 8)
    out, k1, k2, mx = run(dims, block, mul, True, vol, 2, M.BOUNDARY_CIRCULAR)
    ref, _ = O.decon_run(vol[3], vol[0], vol[1], k1, k2, block, 2, mul=mul, lam=0.006, max_intensities=mx)
    assert rel(out, ref) <= 1e-5


def test_mul_tiles_in_slabs_of_two_streams():
    # 288 columns and rows of 230 planes, 76 MB of spectrum: two slabs and more; three views on one psi transform
    dims, kd, block = (256, 250, 230), (21, 21, 41), (128, 128, 192)
    vol = volume(dims, kd, 3, 9)
    assert rel(run(dims, block, True, False, vol)[0], run(dims, block, True, True, vol)[0]) <= 1e-6


def test_steps_with_a_dropped_block_stay_on_the_blocks():
    # the first block's box has no weight in view 0: with the filter on the step runs the blocks that are left
    dims, kd, block = (60, 40, 36), (5, 5, 5), (24, 24, 24)
    vol = volume(dims, kd, 2, 10)
    vol[1][0][:20, :20, :20] = 0.0
    a, k1, k2, mx = run(dims, block, False, False, vol, 2)
    b = run(dims, block, False, True, vol, 2)[0]
    ref, _ = O.decon_run(vol[3], vol[0], vol[1], k1, k2, block, 2, lam=0.006, max_intensities=mx)
    assert rel(a, ref) <= 1e-5 and rel(a, b) <= 2e-6


def test_mul_product_beyond_the_float_range_on_plane_kernels():
    # conv2 of about 1e10 in four views, their product beyond the float range (the separable and row kernels'
    # case is in the parity tests); 1e-5 on the effective region, as there
    b, kd = (128, 128, 64), (5, 5, 7)
    rng = np.random.default_rng(3)
    shape = b[::-1]
    k1s = [synthetic.make_psf(kd, 1.0, 1.5, a) for a in (0.0, 45.0, 90.0, 135.0)]
    k2s = [O.invert_kernel(k) for k in k1s]
    psi = rng.uniform(0.5e-8, 2e-8, shape).astype(np.float32)
    imgs = [rng.uniform(50, 300, shape).astype(np.float32) for _ in range(4)]
    ws = [rng.uniform(0.1, 1, shape).astype(np.float32) for _ in range(4)]
    ref, _ = O.block_mul(psi, imgs, ws, k1s, k2s, 0.006, 1e-4, [300.0] * 4)
    old = os.environ.get("MVR_PLANE_KERNELS")
    os.environ["MVR_PLANE_KERNELS"] = "1"  # read when kernels are set
    try:
        with M.BlockWorker(b, 1e-4, 0.006, 4, M.BOUNDARY_CIRCULAR) as wk:
            for v in range(4):
                wk.set_kernels(v, k1s[v], k2s[v])
            out = psi.copy()
            wk.run_iteration_mul(out, imgs, ws, [300.0] * 4)
    finally:
        if old is None:
            del os.environ["MVR_PLANE_KERNELS"]
        else:
            os.environ["MVR_PLANE_KERNELS"] = old
    sl = tuple(slice(kd[d] - 1, b[d] - kd[d] + 1) for d in (2, 1, 0))
    assert rel(out[sl], ref[sl]) <= 1e-5 and (out[sl] > 1.0).all()


@pytest.mark.parametrize("views", [3, 7, 16])
def test_mul_volume_of_many_views(views):
    dims, kd, block = (40, 33, 28), (5, 5, 5), (24, 24, 24)
    vol = volume(dims, kd, views, views)
    out, k1, k2, mx = run(dims, block, True, False, vol)
    ref, _ = O.decon_run(vol[3], vol[0], vol[1], k1, k2, block, 1, mul=True, lam=0.006, max_intensities=mx)
    assert rel(out, ref) <= 1e-5
