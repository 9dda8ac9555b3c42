"""Iterations without statistics run on the library's own tiles of the volume (separable
transforms, csrc/sep.cuh): every transform length, volumes of more than one tile, odd and even
rows, Seq and Mul, against the oracle driver on the caller's block grid.

Tolerance: relative L2 1e-5 after one iteration (the FP32 bound of one iteration elsewhere), 1e-6
against the same GPU iteration on the caller's blocks (float rounding of two transforms).
"""
import os

import numpy as np
import pytest

import mvrgb300 as M
import oracle as O
import synthetic

pytestmark = pytest.mark.gpu

LEN_X = (64, 96, 128, 160, 192, 224, 256, 288, 320, 384, 448, 512, 576)
LEN_YZ = (32, 48, 64, 80, 96, 112, 128, 144, 160, 192, 224, 256, 288, 320, 360, 400, 432, 480, 576)


def rel(a, b):
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def case(dims, kd, nv, seed):
    rng = np.random.default_rng(seed)
    shape = dims[::-1]
    imgs = [rng.uniform(5, 200, shape).astype(np.float32) for _ in range(nv)]
    for im in imgs:
        im[rng.random(shape) < 0.02] = 0  # voxels without data
    ws = [rng.uniform(0.2, 0.9, shape).astype(np.float32) for _ in range(nv)]
    psfs = [synthetic.make_psf(kd, 1.0, 1.5, 40.0 * v) for v in range(nv)]
    psi = rng.uniform(5, 150, shape).astype(np.float32)
    return imgs, ws, psfs, psi


def run(dims, kd, block, mul, blocks, seed, nv=2, its=1):
    imgs, ws, psfs, psi = case(dims, kd, nv, seed)
    old = os.environ.get("MVR_RATIO_BAND")
    if blocks:
        os.environ["MVR_RATIO_BAND"] = "0"  # keeps the steps on the caller's blocks
    try:
        with M.Deconvolution(dims, nv, block, mul=mul, psf_type=M.PSF_INDEPENDENT, lam=0.006) as d:
            for v in range(nv):
                d.set_view(v, imgs[v], ws[v], psfs[v])
            d.prepare()
            d.set_psi(psi)
            ks = [d.kernels(v, psfs[v].shape) for v in range(nv)]
            mx = d.max_intensities()
            d.run_iterations(its)
            out = d.get_psi()
    finally:
        if blocks:
            if old is None:
                del os.environ["MVR_RATIO_BAND"]
            else:
                os.environ["MVR_RATIO_BAND"] = old
    return out, (psi, imgs, ws, [k[0] for k in ks], [k[1] for k in ks], mx)


def check(dims, kd, block, mul, seed):
    out, (psi, imgs, ws, k1s, k2s, mx) = run(dims, kd, block, mul, False, seed)
    ref, _ = O.decon_run(psi, imgs, ws, k1s, k2s, block, 1, mul=mul, lam=0.006, max_intensities=mx)
    assert np.isfinite(out).all()
    assert rel(out, ref) <= 1e-5
    assert rel(out, run(dims, kd, block, mul, True, seed)[0]) <= 1e-6


@pytest.mark.parametrize("axis,n", [(0, n) for n in LEN_X] + [(a, n) for a in (1, 2) for n in LEN_YZ])
def test_every_length_filled_to_the_last_voxel(axis, n):
    # the volume and the kernel's reach (2 either side) fill the domain of n along one axis
    dims = [37, 26, 22]
    dims[axis] = n - 4
    block = [48, 36, 36]
    block[axis] = 96
    check(tuple(dims), (5, 5, 5), tuple(block), bool((n // 16) % 2), n + axis)


@pytest.mark.parametrize("dims,kd,block,mul", [
    ((573, 26, 22), (5, 5, 5), (96, 36, 36), False),   # one voxel too long for one tile, each axis
    ((38, 573, 22), (5, 7, 5), (48, 96, 36), True),
    ((37, 26, 573), (7, 5, 5), (48, 36, 96), False),
    ((590, 580, 9), (5, 5, 3), (160, 160, 20), False),  # four tiles
    ((8, 9, 7), (3, 5, 7), (20, 20, 28), True),        # smaller than every length
    ((64, 31, 47), (31, 15, 31), (128, 64, 128), False),  # the reach covers half of the volume
    ((16, 8, 16), (31, 15, 31), (64, 32, 64), False),   # reach = size - 1: one reflection still suffices
])
def test_tiles_and_short_volumes(dims, kd, block, mul):
    check(dims, kd, block, mul, sum(dims))


def test_what_stays_on_the_blocks():
    # even kernels, a kernel that reflects twice, a dropped block: the grid decides the result there
    for dims, kd, block in (((36, 30, 44), (4, 6, 5), (40, 40, 40)), ((15, 30, 30), (31, 5, 5), (64, 32, 32))):
        a, _ = run(dims, kd, block, False, False, 3)
        b, _ = run(dims, kd, block, False, True, 3)
        assert rel(a, b) <= 1e-6


def test_unaligned_device_volumes():
    # device images and weights on 4-byte boundaries (no 8-byte loads), even row length
    torch = pytest.importorskip("torch")
    dims, kd, block = (64, 30, 26), (5, 5, 5), (48, 36, 36)
    imgs, ws, psfs, psi = case(dims, kd, 2, 11)
    ref, _ = run(dims, kd, block, False, False, 11)
    n = psi.size
    keep = []
    with M.Deconvolution(dims, 2, block, psf_type=M.PSF_INDEPENDENT, lam=0.006) as d:
        for v in range(2):
            p = []
            for a in (imgs[v], ws[v]):
                t = torch.empty(n + 1, dtype=torch.float32, device="cuda")
                t[1:].copy_(torch.from_numpy(a.reshape(-1)))
                keep.append(t)
                p.append(t[1:].data_ptr())
            torch.cuda.synchronize()
            d.set_view_device(v, p[0], p[1], psfs[v])
        d.prepare()
        d.set_psi(psi)
        d.run_iterations(1)
        out = d.get_psi()
    assert np.array_equal(out, ref)


@pytest.mark.parametrize("b,kd,boundary", [
    ((64, 32, 48), (5, 7, 9), M.BOUNDARY_CIRCULAR),
    ((96, 112, 80), (9, 5, 15), M.BOUNDARY_CIRCULAR),
    ((59, 43, 28), (5, 5, 5), M.BOUNDARY_REFERENCE),   # domain 64 x 48 x 32, filled
    ((60, 45, 29), (5, 5, 5), M.BOUNDARY_REFERENCE),   # one voxel more on every axis
    ((31, 30, 27), (6, 4, 8), M.BOUNDARY_REFERENCE),   # even kernels
])
def test_block_iteration_on_separable_transforms(b, kd, boundary):
    # the whole block and its statistics (reference boundary), the effective region (circular)
    rng = np.random.default_rng(sum(b))
    shape = b[::-1]
    k1 = synthetic.make_psf(kd, 1.0, 1.5, 30.0)
    k2 = O.invert_kernel(k1)
    img = rng.uniform(5, 300, shape).astype(np.float32)
    img[rng.random(shape) < 0.05] = 0
    w = rng.uniform(0, 1, shape).astype(np.float32)
    psi = rng.uniform(5, 300, shape).astype(np.float32)
    ref, ref_st = O.block_seq(psi, img, w, k1, k2, 0.006, 1e-4, 300.0)
    with M.BlockWorker(b, 1e-4, 0.006, 1, boundary) as wk:
        wk.set_kernels(0, k1, k2)
        out = psi.copy()
        st = wk.run_iteration(0, out, img, w, 300.0)
    if boundary == M.BOUNDARY_CIRCULAR:
        e = [k - 1 for k in kd]
        sl = tuple(slice(e[d], b[d] - e[d]) for d in (2, 1, 0))
        assert rel(out[sl], ref[sl]) <= 1e-5
        ch = out.astype(np.float64) - psi
        assert st.sum_change == pytest.approx(float(ch.sum()), rel=1e-4, abs=1e-2)
        assert st.max_change == pytest.approx(float(ch.max()), rel=1e-5)
    else:
        assert rel(out, ref) <= 1e-5
        scale = float(np.abs(out.astype(np.float64) - psi).sum()) + 1.0
        assert abs(st.sum_change - ref_st[0]) <= 1e-4 * scale
        assert abs(st.max_change - ref_st[1]) <= 1e-4 * max(1.0, abs(ref_st[1]))


def test_mul_block_with_one_view_off_the_separable_path():
    # a 21-voxel kernel reflects twice in a block of 8 rows: its view has no separable transforms,
    # and the Mul step of both views runs on the block kernels
    b = (40, 8, 24)
    rng = np.random.default_rng(5)
    shape = b[::-1]
    psi = rng.uniform(5, 300, shape).astype(np.float32)
    imgs = [rng.uniform(5, 300, shape).astype(np.float32) for _ in range(2)]
    ws = [rng.uniform(0, 0.5, shape).astype(np.float32) for _ in range(2)]
    k1s = [synthetic.make_psf(k, 1.0, 1.5, 20.0) for k in ((5, 5, 5), (5, 21, 5))]
    k2s = [O.invert_kernel(k) for k in k1s]
    ref, _ = O.block_mul(psi, imgs, ws, k1s, k2s, 0.006, 1e-4, [300.0, 280.0])
    with M.BlockWorker(b, 1e-4, 0.006, 2, M.BOUNDARY_REFERENCE) as wk:
        for v in range(2):
            wk.set_kernels(v, k1s[v], k2s[v])
        out = psi.copy()
        wk.run_iteration_mul(out, imgs, ws, [300.0, 280.0])
        assert rel(out, ref) <= 1e-5
        one = psi.copy()  # the first view alone keeps its own path
        wk.run_iteration(0, one, imgs[0], ws[0], 300.0)
    r0, _ = O.block_seq(psi, imgs[0], ws[0], k1s[0], k2s[0], 0.006, 1e-4, 300.0)
    assert rel(one, r0) <= 1e-5


def test_mul_block_with_kernels_of_two_sizes():
    b = (40, 36, 24)
    rng = np.random.default_rng(6)
    shape = b[::-1]
    psi = rng.uniform(5, 300, shape).astype(np.float32)
    imgs = [rng.uniform(5, 300, shape).astype(np.float32) for _ in range(3)]
    ws = [rng.uniform(0, 0.4, shape).astype(np.float32) for _ in range(3)]
    k1s = [synthetic.make_psf(k, 1.0, 1.5, 20.0) for k in ((5, 5, 5), (5, 5, 5), (9, 15, 7))]
    k2s = [O.invert_kernel(k) for k in k1s]
    mx = [300.0, 280.0, 260.0]
    ref, _ = O.block_mul(psi, imgs, ws, k1s, k2s, 0.006, 1e-4, mx)
    with M.BlockWorker(b, 1e-4, 0.006, 3, M.BOUNDARY_REFERENCE) as wk:
        for v in range(3):
            wk.set_kernels(v, k1s[v], k2s[v])
        out = psi.copy()
        wk.run_iteration_mul(out, imgs, ws, mx)
    assert rel(out, ref) <= 1e-5


@pytest.mark.parametrize("b,kd", [((59, 43, 28), (5, 5, 5)), ((333, 30, 27), (7, 5, 3))])
def test_queued_iterations_in_place_on_odd_rows(b, kd):
    # psi is read and written by one kernel and read by the next one, launched early; rows of an odd length
    # share 32-byte sectors between CTAs.  Three iterations queued without a wait against the oracle's
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(sum(b))
    shape = b[::-1]
    k1 = synthetic.make_psf(kd, 1.0, 1.5, 30.0)
    k2 = O.invert_kernel(k1)
    img = rng.uniform(5, 300, shape).astype(np.float32)
    w = rng.uniform(0, 1, shape).astype(np.float32)
    ref = rng.uniform(5, 300, shape).astype(np.float32)
    d = [torch.from_numpy(a).cuda() for a in (ref, img, w)]
    torch.cuda.synchronize()
    with M.BlockWorker(b, 1e-4, 0.006, 1, M.BOUNDARY_REFERENCE) as wk:
        wk.set_kernels(0, k1, k2)
        for _ in range(3):
            wk.run_iteration_device(0, *[t.data_ptr() for t in d], 300.0)
        wk.synchronize()
    for _ in range(3):
        ref, _ = O.block_seq(ref, img, w, k1, k2, 0.006, 1e-4, 300.0)
    assert rel(d[0].cpu().numpy(), ref) <= 3e-5  # 1e-5 an iteration, as above


@pytest.mark.parametrize("mul", [False, True])
def test_dim_blocks_far_from_bright_ones(mul):
    # beads of 2e4 in the first 180 columns, 1e-3 to 2e-3 elsewhere: blocks from column 344 on hold no bead, and
    # their voxels (from 352 on) keep the rounding of their own transforms, voxel by voxel; the second view's
    # step reads the first one's 8 columns beyond, so from 360 on.  Tolerance: the FP32 bound of one iteration,
    # here relative to each voxel
    fft = pytest.importorskip("scipy.signal")
    dims, kd, block, nv = (560, 48, 48), (9, 9, 9), (192, 64, 64), 2
    rng = np.random.default_rng(31)
    shape = dims[::-1]
    psi = rng.uniform(1e-3, 2e-3, shape).astype(np.float32)
    psi[rng.integers(0, 48, 30), rng.integers(0, 48, 30), rng.integers(0, 180, 30)] = 2e4
    psfs = [synthetic.make_psf(kd, 1.0, 1.5, 40.0 * v) for v in range(nv)]
    imgs = [np.maximum(fft.fftconvolve(psi[:, :, :200].astype(np.float64), p.astype(np.float64), "same"), 1e-3) for p in psfs]
    imgs = [np.concatenate([i, fft.fftconvolve(psi[:, :, 200:].astype(np.float64), p.astype(np.float64), "same")], 2)
            for i, p in zip(imgs, psfs)]
    imgs = [(i * rng.uniform(0.7, 1.4, shape)).astype(np.float32) for i in imgs]
    ws = [rng.uniform(0.2, 0.5, shape).astype(np.float32) for _ in range(nv)]
    with M.Deconvolution(dims, nv, block, mul=mul, psf_type=M.PSF_INDEPENDENT, lam=0.006) as d:
        for v in range(nv):
            d.set_view(v, imgs[v], ws[v], psfs[v])
        d.prepare()
        d.set_psi(psi)
        ks = [d.kernels(v, psfs[v].shape) for v in range(nv)]
        mx = d.max_intensities()
        d.run_iterations(1)
        out = d.get_psi()
    ref, _ = O.decon_run(psi, imgs, ws, [k[0] for k in ks], [k[1] for k in ks], block, 1, mul=mul, lam=0.006,
                         max_intensities=mx, fp64=True)
    assert rel(out, ref) <= 1e-5
    dark = np.s_[:, :, 360:]
    assert ref[dark].max() < 0.1
    assert np.abs(out[dark] / ref[dark] - 1).max() <= 1e-5


@pytest.mark.parametrize("mul", [False, True])
def test_dim_block_beside_bright_voxels_it_does_not_read(mul):
    # beads of 2e4 in columns 364 to 387 alone: the block of [176, 352) reads [168, 360), its domain of 224 would
    # reach to column 392.  Voxels below 344 (the second view's step reads the first one's 8 columns beyond) keep
    # the rounding of their own transforms.  Tolerance as above
    fft = pytest.importorskip("scipy.signal")
    dims, kd, block, nv = (560, 48, 48), (9, 9, 9), (192, 64, 64), 2
    rng = np.random.default_rng(37)
    shape = dims[::-1]
    psi = rng.uniform(1e-3, 2e-3, shape).astype(np.float32)
    psi[rng.integers(0, 48, 30), rng.integers(0, 48, 30), rng.integers(364, 388, 30)] = 2e4
    psfs = [synthetic.make_psf(kd, 1.0, 1.5, 40.0 * v) for v in range(nv)]
    imgs = [np.maximum(fft.fftconvolve(psi.astype(np.float64), p.astype(np.float64), "same"), 1e-3) for p in psfs]
    imgs = [(i * rng.uniform(0.7, 1.4, shape)).astype(np.float32) for i in imgs]
    ws = [rng.uniform(0.2, 0.5, shape).astype(np.float32) for _ in range(nv)]
    with M.Deconvolution(dims, nv, block, mul=mul, psf_type=M.PSF_INDEPENDENT, lam=0.006) as d:
        for v in range(nv):
            d.set_view(v, imgs[v], ws[v], psfs[v])
        d.prepare()
        d.set_psi(psi)
        ks = [d.kernels(v, psfs[v].shape) for v in range(nv)]
        mx = d.max_intensities()
        d.run_iterations(1)
        out = d.get_psi()
    ref, _ = O.decon_run(psi, imgs, ws, [k[0] for k in ks], [k[1] for k in ks], block, 1, mul=mul, lam=0.006,
                         max_intensities=mx, fp64=True)
    assert rel(out, ref) <= 1e-5
    assert ref[:, :, :344].max() < 0.1
    assert np.abs(out[:, :, :344] / ref[:, :, :344] - 1).max() <= 1e-5


def test_quotient_by_a_value_above_2_to_126():
    # a hot voxel of 1.2e38, a kernel of one voxel: the quotient 1e38 / 1.2e38 (the approximate division alone
    # returns 0 there), psi becomes 1e38.  A periodic domain: an extended one can hold mirror images of the
    # voxel, and the transform's sum of those leaves the float range
    b = (64, 32, 32)
    psi = np.ones(b[::-1], np.float32)
    img = np.zeros(b[::-1], np.float32)  # quotient 1
    psi[9, 10, 20], img[9, 10, 20] = 1.2e38, 1e38
    w = np.ones_like(psi)
    one = np.ones((1, 1, 1), np.float32)
    with M.BlockWorker(b, 1e-4, 0.0, 1, M.BOUNDARY_CIRCULAR) as wk:
        wk.set_kernels(0, one, one)
        wk.run_iteration(0, psi, img, w, 1e38)
    assert abs(psi[9, 10, 20] / 1e38 - 1) <= 1e-5
