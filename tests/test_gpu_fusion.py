"""GPU input preparation (ProcessInputImages.fuseGroups for one group) against the CPU
restatement: affine-transformed views with linear interpolation, cosine blending, weighted
average and summed deconvolution weights.  Tolerance: 1e-5 relative on the fused image
(float interpolation), 1e-6 on the weights; voxels whose sample falls within 1e-9 of a
view's border (where double rounding may decide inside / outside) are excluded."""
import math

import numpy as np
import pytest

import mvrgb300 as M
import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def model(angle_deg, scale_z, t):
    a = math.radians(angle_deg)
    R = np.array([[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]])
    S = np.diag([1.0, 1.0, scale_z])
    return np.hstack([R @ S, np.asarray(t, dtype=np.float64).reshape(3, 1)])


@pytest.mark.parametrize("blend", [False, True])
def test_fuse_group_matches_oracle(blend):
    rng = np.random.default_rng(7)
    views = []
    for k, (ang, tz) in enumerate([(0.0, 0.0), (33.0, 4.0), (-61.0, -3.0)]):
        img = rng.uniform(0, 300, (20, 40, 48)).astype(np.float32)  # [z][y][x]
        m = model(ang, 1.5, (2.37 + k, -1.71, tz + 0.43))  # fractional: samples rarely land on a border
        v = {"img": img, "model": m}
        if k == 1:
            v["intensity"] = (1.37, -4.25)  # IntensityAdjuster of the second view
        if blend:
            v["fusion"] = ((2.0, 2.0, 1.0), (10.0, 10.0, 4.0))
            v["decon"] = ((1.0, 1.0, 0.5), (6.0, 6.0, 3.0))
        views.append(v)
    bb_min, bb_dims = (-10, -6, -14), (64, 44, 40)
    ref_img, ref_w = O.fuse_group(views, bb_min, bb_dims)
    dev = [torch.from_numpy(v["img"]).cuda() for v in views]
    out_i = torch.empty((bb_dims[2], bb_dims[1], bb_dims[0]), dtype=torch.float32, device="cuda")
    out_w = torch.empty_like(out_i)
    gv = []
    for v, d in zip(views, dev):
        g = {"img_ptr": d.data_ptr(), "dims": (v["img"].shape[2], v["img"].shape[1], v["img"].shape[0]),
             "model": v["model"], "intensity": v.get("intensity")}
        if blend:
            g["fusion"], g["decon"] = v["fusion"], v["decon"]
        gv.append(g)
    M.fuse_group(gv, bb_min, bb_dims, out_i.data_ptr(), out_w.data_ptr())
    img, w = out_i.cpu().numpy(), out_w.cpu().numpy()
    # voxels far from every view's border decision
    z, y, x = np.meshgrid(*[np.arange(n) for n in bb_dims[::-1]], indexing="ij")
    s = np.stack([x + bb_min[0], y + bb_min[1], z + bb_min[2]], -1).astype(np.float64)
    safe = np.ones(s.shape[:-1], bool)
    for v in views:
        inv = O._invert_affine(v["model"])
        t = s @ inv[:, :3].T + inv[:, 3]
        dims = np.array(v["img"].shape[::-1], dtype=np.float64)
        safe &= np.all((np.abs(t) > 1e-9) & (np.abs(t - (dims - 1)) > 1e-9), axis=-1)
    assert safe.mean() > 0.99
    assert np.abs(img - ref_img)[safe].max() <= 1e-5 * max(1.0, float(np.abs(ref_img).max()))
    assert np.abs(w - ref_w)[safe].max() <= 1e-6
    assert (ref_img > 0).mean() > 0.3  # the views cover a good part of the box


@pytest.mark.parametrize("bb_min,bb_dims,angle,scale,shift,nv,blend", [
    ((0, 0, 0), (1, 1, 1), 10.0, 1.0, (-3.3, -2.7, -1.9), 1, False),       # one voxel
    ((2, 1, 1), (7, 9, 3), 25.0, 1.5, (0.31, -0.47, 0.23), 2, True),       # a row group and one row more
    ((-3, -2, -1), (33, 8, 5), 0.0, 1.0, (0.0, 0.0, 0.0), 1, True),        # samples on the voxels and borders
    ((-3, -2, -9), (40, 17, 30), 90.0, 1.0, (0.0, 0.0, 8.0), 1, False),    # axes exchanged
    ((1000000, -2000000, 500000), (31, 20, 9), 33.0, 2.0, (1000000.37, -2000000.61, 500000.43), 3, True),  # far away
    ((0, 0, 0), (300, 3, 2), -20.0, 1.0, (0.7, 0.1, 0.9), 16, True),       # 16 views, rows longer than a CTA
])
def test_fuse_group_edges(bb_min, bb_dims, angle, scale, shift, nv, blend):
    # the pair arithmetic against the oracle's doubles; voxels within 1e-6 of a border or of a step of the
    # blending table (1 / 1000 of the range) may round to the other side and are left out
    rng = np.random.default_rng(nv + bb_dims[0])
    views = []
    for k in range(nv):
        img = rng.uniform(0, 300, (8, 24, 40)).astype(np.float32)
        v = {"img": img, "model": model(angle + 3.0 * k, scale, np.asarray(shift) + 0.11 * k)}
        if k % 3 == 1:
            v["intensity"] = (0.731, 12.5)
        if blend:
            v["fusion"] = ((1.0, 2.0, 0.0), (10.0, 7.0, 3.0))
            v["decon"] = ((0.5, 0.0, 0.5), (6.0, 6.0, 2.0))
        views.append(v)
    ref_img, ref_w = O.fuse_group(views, bb_min, bb_dims)
    dev = [torch.from_numpy(v["img"]).cuda() for v in views]
    out_i = torch.full((bb_dims[2], bb_dims[1], bb_dims[0]), -1.0, device="cuda")
    out_w = torch.full_like(out_i, -1.0)
    gv = [dict(v, img_ptr=d.data_ptr(), dims=(40, 24, 8)) for v, d in zip(views, dev)]
    M.fuse_group(gv, bb_min, bb_dims, out_i.data_ptr(), out_w.data_ptr())
    z, y, x = np.meshgrid(*[np.arange(n) for n in bb_dims[::-1]], indexing="ij")
    s = np.stack([x + bb_min[0], y + bb_min[1], z + bb_min[2]], -1).astype(np.float64)
    safe = np.ones(s.shape[:-1], bool)
    dims = np.array((40, 24, 8), dtype=np.float64)
    for v in views:
        inv = O._invert_affine(v["model"])
        t = s @ inv[:, :3].T + inv[:, 3]
        whole = np.abs(t - np.round(t)) == 0  # exact samples take the same branch on both sides
        near = (np.abs(t) <= 1e-6) | (np.abs(t - (dims - 1)) <= 1e-6)
        safe &= ~np.any(near & ~whole, axis=-1)
        for key in ("fusion", "decon"):
            if v.get(key):
                b, r = (np.asarray(a) for a in v[key])
                e = np.minimum(t - b, dims - 1 - t - b) / r * 1000 + 0.5
                safe &= ~np.any((np.abs(e - np.round(e)) < 1e-3) & (e > 0) & (e < 1001), axis=-1)
    got_i, got_w = out_i.cpu().numpy(), out_w.cpu().numpy()
    assert safe.mean() > (0.8 if nv < 16 else 0.3) or angle == 0.0
    assert np.abs(got_i - ref_img)[safe].max(initial=0.0) <= 1e-5 * max(1.0, float(np.abs(ref_img).max()))
    assert np.abs(got_w - ref_w)[safe].max(initial=0.0) <= 1e-6 * max(1, nv)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.3e38, -3.3e38])
@pytest.mark.parametrize("nv,intensity", [(1, None), (3, None), (1, (1.5, -2.0)), (2, (-4.0, 0.0))])
def test_fuse_group_samples_beyond_the_float_range(value, nv, intensity):
    # samples that are infinite, not a number, or so large that differences and sums leave the float range:
    # the double sums of the oracle.  Where it says NaN (Inf - Inf, or a NaN sample), max(1, NaN) is 1 here;
    # that changes a voxel of one view only, so voxels of several are left out there
    rng = np.random.default_rng(3)
    views = []
    for k in range(nv):
        img = rng.uniform(1, 300, (9, 16, 24)).astype(np.float32)
        img[3:5, 4:9, 6 + k:12 + k] = value
        img[5, 10, 7:9] = (value, -value)
        v = {"img": img, "model": model(21.0 + 9 * k, 1.25, (0.37 + k, -0.71, 0.43))}
        if intensity:
            v["intensity"] = intensity
        v["fusion"] = v["decon"] = ((0.0, 0.0, 0.0), (6.0, 6.0, 3.0))
        views.append(v)
    bb_min, bb_dims = (-2, -1, -9), (30, 18, 24)
    with np.errstate(all="ignore"):
        ref_img, ref_w = O.fuse_group(views, bb_min, bb_dims)
    dev = [torch.from_numpy(v["img"]).cuda() for v in views]
    out = [torch.full((bb_dims[2], bb_dims[1], bb_dims[0]), -1.0, device="cuda") for _ in range(2)]
    M.fuse_group([dict(v, img_ptr=d.data_ptr(), dims=(24, 16, 9)) for v, d in zip(views, dev)], bb_min, bb_dims,
                 out[0].data_ptr(), out[1].data_ptr())
    img, w = (o.cpu().numpy() for o in out)
    nan = np.isnan(ref_img)
    if nv == 1:
        ref_img = np.where(nan, np.float32(1), ref_img)
        nan[:] = False
    assert not np.isnan(img).any()
    odd = np.abs(ref_img) > 1e30
    assert odd.any() or not value > 0 or intensity == (-4.0, 0.0)
    same = np.isinf(ref_img) & ~nan
    assert np.array_equal(img[same], ref_img[same])
    fin = np.isfinite(ref_img)
    assert np.abs(img / np.where(fin, ref_img, 1) - 1)[fin & (ref_img != 0)].max() <= 1e-5
    assert not img[fin & (ref_img == 0)].any()
    assert np.abs(w - ref_w).max() <= 1e-6 * nv


def test_fuse_group_next_to_bright_samples():
    # a dim sample whose bright neighbour has a weight of 2e-5 to 3e-4: the weights' relative error counts,
    # not their distance to 1.  Three interpolations of two rounded weights, a product and a sum each, and
    # the oracle's eight rounded terms: 1.1e-6
    rng = np.random.default_rng(11)
    for frac in (2e-5, 3e-4, 1 - 1e-4):
        img = np.where(rng.random((10, 14, 30)) < 0.3, rng.uniform(1e6, 4e6, (10, 14, 30)), rng.uniform(1, 3, (10, 14, 30)))
        img = img.astype(np.float32)
        v = {"img": img, "model": model(0.0, 1.0, (-frac, frac - 1.0, -frac))}
        bb_min, bb_dims = (1, 1, 1), (26, 10, 7)
        ref, _ = O.fuse_group([v], bb_min, bb_dims)
        d = torch.from_numpy(img).cuda()
        out = [torch.full((bb_dims[2], bb_dims[1], bb_dims[0]), -1.0, device="cuda") for _ in range(2)]
        M.fuse_group([dict(v, img_ptr=d.data_ptr(), dims=(30, 14, 10))], bb_min, bb_dims, out[0].data_ptr(), out[1].data_ptr())
        assert (ref > 0).all()
        assert np.abs(out[0].cpu().numpy() / ref - 1).max() <= 2e-6


def test_fuse_group_rows_beyond_the_float_integers():
    # a box of one row of 2^24 + 60 voxels: the end of the row, where x is no float any more, equals a small
    # box there (the oracle's)
    rng = np.random.default_rng(2)
    n = 1 << 24
    img = rng.uniform(1, 300, (6, 9, 50)).astype(np.float32)
    v = {"img": img, "model": model(0.0, 1.0, (n + 3.37, -2.21, -1.63)), "fusion": ((0, 0, 0), (5, 5, 5)),
         "decon": ((0, 0, 0), (4, 4, 4))}
    ref = O.fuse_group([v], (n, 0, 0), (60, 1, 1))
    d = torch.from_numpy(img).cuda()
    out = [torch.full((n + 60,), -1.0, device="cuda") for _ in range(2)]
    M.fuse_group([dict(v, img_ptr=d.data_ptr(), dims=(50, 9, 6))], (0, 0, 0), (n + 60, 1, 1), out[0].data_ptr(), out[1].data_ptr())
    for a, b in zip(out, ref):
        assert np.abs(a[n:].cpu().numpy() - b.reshape(-1)).max() <= 1e-5 * b.max()
        assert not a[:n].any()
