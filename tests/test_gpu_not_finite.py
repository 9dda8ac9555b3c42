"""Values that are not finite, in psi or in a quotient, reach the blocks that read them and no other: on
the caller's block grid through the blocks' transforms, on the library's tiles through the marks of the
blocks (BadMap, csrc/kernels.cuh).  Against the oracle driver, whose blocks are transforms of their own;
tolerance per voxel: 1e-5 of the volume's range and an iteration, the FP32 bound of one iteration elsewhere
(FP64: the rounding of psi to float, in which it is read back)."""
import os

import numpy as np
import pytest

import mvrgb300 as M
import oracle as O
import synthetic

pytestmark = pytest.mark.gpu


def case(dims, kd, nv, seed):
    rng = np.random.default_rng(seed)
    shape = dims[::-1]
    imgs = [rng.uniform(5, 200, shape).astype(np.float32) for _ in range(nv)]
    ws = [rng.uniform(0.2, 0.9, shape).astype(np.float32) for _ in range(nv)]
    psfs = [synthetic.make_psf(kd, 1.0, 1.5, 40.0 * v) for v in range(nv)]
    return imgs, ws, psfs, rng.uniform(5, 150, shape).astype(np.float32)


def run(dims, block, mul, fp64, its, imgs, ws, psfs, psi, bad_imgs, blocks=False):
    old = os.environ.get("MVR_RATIO_BAND")
    if blocks:
        os.environ["MVR_RATIO_BAND"] = "0"  # keeps the steps on the caller's blocks
    try:
        with M.Deconvolution(dims, len(imgs), block, mul=mul, psf_type=M.PSF_INDEPENDENT, lam=0.006,
                             precision=M.PRECISION_FP64 if fp64 else M.PRECISION_FP32) as d:
            for v in range(len(imgs)):
                d.set_view(v, imgs[v], ws[v], psfs[v])
            d.prepare()
            d.set_psi(psi)
            for v in range(len(imgs)):
                d.update_images(v, bad_imgs[v], ws[v])
            ks = [d.kernels(v, psfs[v].shape) for v in range(len(imgs))]
            mx = d.max_intensities()
            d.run_iterations(its)
            return d.get_psi(), ks, mx
    finally:
        if blocks:
            if old is None:
                del os.environ["MVR_RATIO_BAND"]
            else:
                os.environ["MVR_RATIO_BAND"] = old


def same(a, b, tol):
    assert np.array_equal(np.isnan(a), np.isnan(b))
    ok = np.isfinite(b)
    assert np.abs(a[ok].astype(np.float64) - b[ok]).max() <= tol * np.abs(b[ok]).max()


@pytest.mark.parametrize("mul", [False, True])
@pytest.mark.parametrize("fp64", [False, True])
@pytest.mark.parametrize("where", ["image", "image at a face", "psi", "psi at a corner", "psi without data", "none"])
def test_blocks_that_read_it_and_no_other(where, mul, fp64):
    # 5 x 3 x 3 blocks of 24^3 on one tile; two iterations, so that marks of the first are gone in the second
    dims, kd, block = (70, 44, 40), (5, 5, 5), (24, 24, 24)
    imgs, ws, psfs, psi = case(dims, kd, 2, 17)
    clean, bad = psi.copy(), [a.copy() for a in imgs]
    at = {"image": (21, 18, 35), "image at a face": (39, 2, 17), "psi": (9, 33, 40), "psi at a corner": (0, 43, 69),
          "psi without data": (12, 20, 66), "none": (0, 0, 0)}[where]
    if where.startswith("image"):
        bad[0][at] = np.inf
        bad[1][1, 1, 1] = np.nan  # not > 0: quotient 1
    elif where.startswith("psi"):
        psi[at] = np.inf if where == "psi" else np.nan
    if where == "psi without data":  # no positive voxel in the last blocks along x: their quotients stay 1
        for a in bad:
            a[:, :, 40:] = 0
    out, ks, mx = run(dims, block, mul, fp64, 2, imgs, ws, psfs, psi, bad)
    with np.errstate(all="ignore"):
        ref, _ = O.decon_run(psi, bad, ws, [k[0] for k in ks], [k[1] for k in ks], block, 2, mul=mul, lam=0.006,
                             max_intensities=mx, fp64=fp64)
        clean, _ = O.decon_run(clean, imgs if "data" not in where else bad, ws, [k[0] for k in ks], [k[1] for k in ks], block,
                               2, mul=mul, lam=0.006, max_intensities=mx, fp64=fp64)
    changed = int((~(np.abs(ref - clean) <= 1e-3 * clean)).sum())
    assert changed <= 1 if where in ("psi without data", "none") else 12 ** 3 <= changed < ref.size // 2
    same(out, ref, 2.0 ** -24 if fp64 else 2e-5)


@pytest.mark.parametrize("mul", [False, True])
def test_tiles_of_two_launches(mul):
    # 20 tiles of 576 x 576 x 32, twelve to a launch: the second launch's tiles, and marks across launches
    dims, kd, block = (2300, 1750, 9), (5, 5, 3), (160, 160, 20)
    imgs, ws, psfs, psi = case(dims, kd, 2, 23)
    for values in ("finite", "not"):
        bad = [a.copy() for a in imgs]
        if values == "not":
            bad[1][4, 1720, 2290] = np.inf
            bad[0][0, 566, 1134] = np.inf  # where four tiles meet
            psi[8, 20, 1600] = np.inf
        a = run(dims, block, mul, False, 1, imgs, ws, psfs, psi, bad)[0]
        b = run(dims, block, mul, False, 1, imgs, ws, psfs, psi, bad, blocks=True)[0]
        same(a, b, 1e-5)
