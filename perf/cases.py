"""Performance cases of the deconvolution framework, through its public Python entry points.

What a user's program has this framework do, from the smallest call to the largest:

* ``block``      one block iteration on device buffers (BlockWorker.run_iteration_device), and
  ``block_host`` the per-block plugin call on host arrays (BlockWorker.run_iteration);
* ``volume``     whole-volume iterations on the device followed by a copy of psi
  (Deconvolution.run_iterations, get_psi_device), sequential or multiplicative, FP32 or FP64,
  with one compute block around the volume, a grid of blocks, or one block size per view;
* ``host``       the whole run on host arrays with the next views uploading (run_host);
* ``fuse``       the input preparation of one group of views (fuse_group);
* ``unet_train`` / ``unet_forward``  the learned proposal's network.

Sizes come from the bench's workloads, the tests and the learned proposal's defaults, or are
generic odd ones.  ``exact`` restates every path in 64 bits with torch.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "multiview-reconstruction_gb300")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import mvrgb300 as M  # noqa: E402
import synthetic  # noqa: E402

DEV = "cuda:0"
PSF_TYPES = {"I": M.PSF_OPTIMIZATION_I, "efficient": M.PSF_EFFICIENT_BAYESIAN, "independent": M.PSF_INDEPENDENT}
# U-Net layers (input channels, output channels)
LAYERS = [(16, 16), (16, 32), (32, 64), (96, 32), (48, 16)]


def _volume(name, dims, views, psf, block, iterations, psf_last=None, mul=False, psf_type="I", lam=0.006,
            boundary="circular", weights="hard", fp64=False, kind="volume", effective=0, grid="fixed"):
    """psf: the first view's PSF size; psf_last: the last view's (sizes in between are spread
    evenly).  grid "fixed": `block` for every view; "tight": `effective` voxels plus each view's
    overlap on every axis, the smallest FFT-friendly block; "plane": the same effective blocks in
    the smallest compute blocks of 192 or 256 (z 192, 256 or 288) that hold them."""
    psf_last = psf_last or psf
    c = {"kind": kind, "x": dims[0], "y": dims[1], "z": dims[2], "views": views, "psf_xy": psf[0], "psf_z": psf[2],
         "psf_last_xy": psf_last[0], "psf_last_z": psf_last[2], "block_x": block[0], "block_y": block[1],
         "block_z": block[2], "grid": grid, "effective": effective, "iterations": iterations, "mul": mul, "psf_type": psf_type,
         "lambda": lam, "boundary": boundary, "weights": weights, "fp64": fp64}
    if name:
        c["name"] = name
    return c


def _block(name, kind, block, psf, boundary, lam=0.006):
    c = {"kind": kind, "x": block[0], "y": block[1], "z": block[2], "psf_xy": psf[0], "psf_z": psf[2],
         "boundary": boundary, "lambda": lam}
    if name:
        c["name"] = name
    return c


def _net(name, kind, batch, dims):
    c = {"kind": kind, "batch": batch, "x": dims[0], "y": dims[1], "z": dims[2]}
    if name:
        c["name"] = name
    return c


def _fuse(name, box, views, scale_z, blend):
    c = {"kind": "fuse", "x": box[0], "y": box[1], "z": box[2], "views": views, "scale_z": scale_z, "blend": blend}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one small block (the smoke test's), where launches and latency count
        _block("block_40x36x44", "block", (40, 36, 44), (5, 5, 9), "reference"),
        # the reference boundary on a block without a special FFT size (the parity tests' block)
        _block("block_156x156x124", "block", (156, 156, 124), (15, 15, 31), "reference", lam=0.0),
        # the drop-in plugin call on host arrays, the 192^3 block of the 4-view workload
        _block("block_host_192", "block_host", (192, 192, 192), (31, 31, 61), "circular"),
        # the reference's own CPU case: 2 views, one block around the volume, 10 iterations
        _volume("2view_128x128x64", (128, 128, 64), 2, (15, 15, 31), (192, 192, 128), 10, psf_type="efficient",
                lam=0.0, weights="ones"),
        # an odd-sized volume in multiplicative mode on the reference boundary
        _volume("mul_3view_211x187x143", (211, 187, 143), 3, (15, 15, 31), (96, 96, 112), 2, mul=True,
                boundary="reference"),
        # the FP64 shadow run of a small volume
        _volume("fp64_2view_96x88x72", (96, 88, 72), 2, (9, 9, 15), (64, 64, 64), 2, fp64=True),
        # the bench's workload: 4 views of 256^3, 192^3 blocks
        _volume("4view_256", (256, 256, 256), 4, (31, 31, 61), (192, 192, 192), 1),
        # a time series from host memory: images and weights of the next step upload meanwhile
        _volume("host_2view_256x256x128", (256, 256, 128), 2, (21, 21, 41), (192, 192, 192), 1, kind="host"),
        # the largest: 6 views of 512 x 512 x 256 with a PSF size per view, 128^3 effective blocks
        _volume("6view_512x512x256", (512, 512, 256), 6, (21, 21, 41), (0, 0, 0), 1, psf_last=(41, 41, 81),
                effective=128, grid="plane"),
        # the input preparation of one group: 3 rotated, anisotropic views into a 256^3 box
        _fuse("fuse_3view_256", (256, 256, 256), 3, 2.5, True),
        # the learned proposal: a training step on 4 crops of 64^3, and its 128^3 coarse grid
        _net("unet_train_4x64", "unet_train", 4, (64, 64, 64)),
        _net("unet_forward_128", "unet_forward", 1, (128, 128, 128)),
    ]


# ---- drawn cases ------------------------------------------------------------------------

def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, lo, hi):
    return 2 * rng.randint(lo // 2, (hi - 1) // 2) + 1


def _friendly(n, even):
    while True:
        k = n
        for r in (2, 3, 5, 7, 11, 13):
            while k % r == 0:
                k //= r
        if k == 1 and not (even and n % 2):
            return n
        n += 1


def _draw_volume(rng, kind):
    while True:
        c = _draw_volume_once(rng, kind)
        cost = 0.0  # voxels through the FFTs of one pass
        for b, k in zip(_blocks(c), _psf_sizes(c)):
            e = [c["effective"] or b[d] - 2 * (k[d] - 1) for d in range(3)]
            count = math.prod(-(-(c["x"], c["y"], c["z"])[d] // e[d]) for d in range(3))
            pad = [b[d] + (k[d] - 1 if c["boundary"] == "reference" else 0) for d in range(3)]
            cost += c["iterations"] * count * math.prod(pad)
        if cost * (12 if c["fp64"] else 2 if c["boundary"] == "reference" else 1) <= 1.2e9:
            return c


def _draw_volume_once(rng, kind):
    fp64 = kind == "volume" and rng.random() < 0.1
    most = 1.5e6 if fp64 else (1.2e7 if kind == "host" else 6.5e7)  # voxels
    while True:
        kxy, kz = _odd(rng, 7, 41), _odd(rng, 9, 81)
        dims = [_logint(rng, 48, 512), _logint(rng, 48, 512), _logint(rng, 40, 400)]
        views = rng.randint(1, 6 if kind == "volume" else 3)
        n = dims[0] * dims[1] * dims[2]
        if n <= most and n * views <= 3e8 and kxy < min(dims[:2]) and kz < dims[2] and kz >= kxy:
            break
    mul = kind == "volume" and not fp64 and rng.random() < 0.25
    last = (kxy, kz)
    if not mul and views > 1 and rng.random() < 0.3:  # a PSF size per view
        last = (_odd(rng, 7, kxy), _odd(rng, 9, kz))
    # every block keeps at least k - 1 effective voxels, as users choose them
    need = [2 * (k - 1) + max(k - 1, 32) for k in (kxy, kxy, kz)]
    fixed = [b for b in ((128, 128, 64), (128, 128, 128), (192, 192, 128), (192, 192, 192), (256, 256, 256))
             if all(b[d] >= need[d] for d in range(3))]
    one = [_friendly(dims[d] + 2 * ((kxy, kxy, kz)[d] - 1), d == 0) for d in range(3)]
    mode = rng.choice(["one", "fixed", "tight", "plane"])
    block, effective, grid = (0, 0, 0), 0, "fixed"
    if mode == "one" and one[0] * one[1] * one[2] <= 4e7:
        block = one
    elif mode in ("one", "fixed") and fixed:
        block = rng.choice(fixed)
    else:
        effective = rng.choice([e for e in (64, 96, 128) if e >= max(kxy, kz) - 1])
        plane = mode == "plane" and effective + 2 * (kz - 1) <= 288
        grid = "plane" if plane else "tight"
    its = rng.choice([1, 2, 5, 10]) if n * views < 1e7 else 1
    return _volume(None, dims, views, (kxy, kxy, kz), block, its, psf_last=(last[0], last[0], last[1]), mul=mul,
                   psf_type=rng.choice(["I", "I", "efficient", "independent"]), lam=rng.choice([0.006, 0.006, 0.0]),
                   boundary="reference" if rng.random() < 0.2 else "circular", weights=rng.choice(["hard", "hard", "ones"]),
                   fp64=fp64, kind=kind, effective=effective, grid=grid)


def draw(rng):
    kind = rng.choice(["volume"] * 7 + ["host", "block", "block", "block_host", "fuse", "unet_train", "unet_forward"])
    if kind in ("volume", "host"):
        return _draw_volume(rng, kind)
    if kind in ("block", "block_host"):
        boundary = rng.choice(["reference", "circular"])
        while True:
            b = [_logint(rng, 24, 256) for _ in range(3)]
            if boundary == "circular":
                b = [_friendly(b[d], d == 0) for d in range(3)]
            k = (_odd(rng, 5, 31), _odd(rng, 5, 61))
            if k[0] <= min(b[:2]) and k[1] <= b[2] and b[0] * b[1] * b[2] <= 1.2e7:
                return _block(None, kind, b, (k[0], k[0], k[1]), boundary, rng.choice([0.006, 0.0]))
    if kind == "fuse":
        return _fuse(None, [_logint(rng, 60, 300) for _ in range(3)], rng.randint(1, 4), rng.choice([1.0, 2.5, 4.0]),
                     rng.random() < 0.75)
    batch = rng.choice([1, 2, 4, 8]) if kind == "unet_train" else 1
    return _net(None, kind, batch, [4 * _logint(rng, 8, 18 if kind == "unet_train" else 36) for _ in range(3)])


# ---- inputs -----------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rand(g, shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=g, device=DEV) * (hi - lo) + lo


def _object(g, shape):
    """Gaussian beads (sigma 1.5) on a smooth body of intensity about 50."""
    n = shape[0] * shape[1] * shape[2]
    beads = torch.zeros(shape, device=DEV)
    count = max(8, n // 80000)
    at = torch.randint(0, n, (count,), generator=g, device=DEV)
    beads.view(-1).index_add_(0, at, _rand(g, (count,), 100.0, 1000.0) * (2 * math.pi * 1.5 ** 2) ** 1.5)
    f = [torch.fft.fftfreq(s, device=DEV) for s in shape[:2]] + [torch.fft.rfftfreq(shape[2], device=DEV)]
    f2 = f[0].view(-1, 1, 1) ** 2 + f[1].view(1, -1, 1) ** 2 + f[2].view(1, 1, -1) ** 2
    spec = torch.fft.rfftn(beads) * torch.exp(-2 * math.pi ** 2 * 1.5 ** 2 * f2)
    obj = torch.fft.irfftn(spec, s=shape)
    r = sum(((torch.arange(s, device=DEV) - (s - 1) / 2) / (0.35 * s)).view([-1 if d == e else 1 for e in range(3)]) ** 2
            for d, s in enumerate(shape))
    return obj.clamp_(min=0) + 50.0 * torch.sigmoid((1.0 - r.sqrt()) * 12.0)


def _conv(vol, k, dtype):
    """Linear convolution of a [z][y][x] volume with a kernel of odd sizes (centre k // 2): the
    valid part."""
    s = [_friendly(n, True) for n in vol.shape]
    f = torch.fft.rfftn(vol.to(dtype), s=s)
    f *= torch.fft.rfftn(k.to(dtype), s=s)
    out = torch.fft.irfftn(f, s=s)
    return out[k.shape[0] - 1:vol.shape[0], k.shape[1] - 1:vol.shape[1], k.shape[2] - 1:vol.shape[2]]


def _mirror(vol, r):
    """Mirror-single extension by r = (z, y, x) voxels on both sides."""
    for d in range(3):
        n = vol.shape[d]
        i = torch.arange(-r[d], n + r[d], device=vol.device)
        i = i.remainder(max(1, 2 * n - 2))
        vol = vol.index_select(d, torch.where(i >= n, 2 * n - 2 - i, i))
    return vol


def _psf_sizes(c):
    v, a, b = c["views"], (c["psf_xy"], c["psf_z"]), (c["psf_last_xy"], c["psf_last_z"])

    def at(i, d):
        t = i / max(1, v - 1)
        return 2 * int(round(((1 - t) * a[d] + t * b[d] - 1) / 2)) + 1

    return [(at(i, 0), at(i, 0), at(i, 1)) for i in range(v)]


def _psfs(sizes):
    """Rotated anisotropic PSFs with side lobes, sigma growing with the box as the bench's do."""
    return [synthetic.make_psf(s, min(1.5, s[0] / 8), min(4.5, s[2] / 7), 180.0 * i / len(sizes), side_lobes=True)
            for i, s in enumerate(sizes)]


def _views(c, seed):
    """Images (Poisson counts of the blurred object over a background of 10), raw weights,
    PSFs and a psi in the middle of a run."""
    g = _gen(seed)
    shape = (c["z"], c["y"], c["x"])
    obj = _object(g, shape)
    psfs = _psfs(_psf_sizes(c))
    imgs, ws = [], []
    for v, p in enumerate(psfs):
        k = torch.from_numpy(p).to(DEV)
        b = _conv(_mirror(obj, [s // 2 for s in k.shape]), k, torch.float32) + 10.0
        imgs.append(torch.poisson(b.clamp_(min=0), generator=g).clamp_(min=1.0).contiguous())
        if c["weights"] == "ones":
            ws.append(torch.ones(shape, device=DEV))
        else:
            ws.append(synthetic._cosine_weight_torch((c["x"], c["y"], c["z"]), 180.0 * v / c["views"], DEV))
    psi = (obj * _rand(g, shape, 0.6, 1.2) + _rand(g, shape, 5.0, 12.0)).contiguous()
    return imgs, ws, psfs, psi


def _blocks(c):
    """Compute block per view."""
    if c["grid"] == "fixed":
        return [(c["block_x"], c["block_y"], c["block_z"])] * c["views"]
    need = [[c["effective"] + 2 * (k[d] - 1) for d in range(3)] for k in _psf_sizes(c)]
    if c["grid"] == "tight":
        return [tuple(_friendly(n[d], d == 0) for d in range(3)) for n in need]
    sizes = [(192, 256), (192, 256), (192, 256, 288)]
    return [tuple(min(p for p in sizes[d] if p >= n[d]) for d in range(3)) for n in need]


def _decon(c, seed):
    imgs, ws, psfs, psi = _views(c, seed)
    blocks = _blocks(c)
    d = M.Deconvolution((c["x"], c["y"], c["z"]), c["views"], blocks[0], mul=c["mul"], psf_type=PSF_TYPES[c["psf_type"]],
                        lam=c["lambda"], boundary=M.BOUNDARY_REFERENCE if c["boundary"] == "reference" else M.BOUNDARY_CIRCULAR,
                        precision=M.PRECISION_FP64 if c["fp64"] else M.PRECISION_FP32,
                        weight_norm=M.WEIGHTS_AS_GIVEN if c["weights"] == "ones" else M.WEIGHTS_HARD)
    for v in range(c["views"]):
        if blocks[v] != blocks[0]:
            d.set_view_block_size(v, blocks[v])
    if c["grid"] == "plane":
        d.set_effective_block_size(-1, (c["effective"],) * 3)
    return d, imgs, ws, psfs, psi


def _block_inputs(c, seed):
    g = _gen(seed)
    shape = (c["z"], c["y"], c["x"])
    k1 = _psfs([(c["psf_xy"], c["psf_xy"], c["psf_z"])] * 2)[1]
    k2 = np.ascontiguousarray(k1[::-1, ::-1, ::-1])
    img = _rand(g, shape, 5.0, 300.0)
    img[_rand(g, shape) < 0.05] = 0.0  # voxels without data
    return k1, k2, img, _rand(g, shape), _rand(g, shape, 5.0, 200.0)


def _fuse_inputs(c, seed):
    g = _gen(seed)
    box = (c["x"], c["y"], c["z"])
    views = []
    for k in range(c["views"]):
        a = math.radians(37.0 * k)
        dims = (box[0], box[1], max(8, int(round(box[2] / c["scale_z"]))))
        rot = np.array([[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]])
        m = rot @ np.diag([1.0, 1.0, c["scale_z"]])
        # the view's centre on the box's centre, a fraction of a voxel off
        t = np.array(box) / 2 - m @ (np.array(dims) / 2) + (0.37 + 0.11 * k, -0.71, 0.43)
        v = {"img": _rand(g, (dims[2], dims[1], dims[0]), 0.0, 300.0), "dims": dims,
             "model": np.hstack([m, t.reshape(3, 1)])}
        if c["blend"]:
            v["fusion"] = ((2.0, 2.0, 1.0), (40.0, 40.0, 15.0))
            v["decon"] = ((1.0, 1.0, 0.5), (12.0, 12.0, 5.0))
        views.append(v)
    return views, box


def _net_inputs(c, seed):
    g = _gen(seed)
    shape = (c["batch"], c["z"], c["y"], c["x"])
    psi = torch.stack([_object(g, shape[1:]) for _ in range(c["batch"])]) + 8.0
    nxt = psi * _rand(g, shape, 0.9, 1.12)
    tgt = nxt * (nxt / psi) * _rand(g, shape, 0.97, 1.03)
    return psi.contiguous(), nxt.contiguous(), tgt.contiguous()


def prepare(case, seed):
    c = case
    s = {"case": c}
    if c["kind"] in ("volume", "host"):
        d, imgs, ws, psfs, psi = _decon(c, seed)
        if c["kind"] == "volume":
            torch.cuda.synchronize()
            for v in range(c["views"]):
                d.set_view_device(v, imgs[v].data_ptr(), ws[v].data_ptr(), psfs[v])
            d.prepare()
            d.set_psi_device(psi.data_ptr())
            s.update(decon=d, keep=(imgs, ws, psi), out=torch.empty_like(psi))
        else:
            h = [[a.cpu().pin_memory().numpy() for a in x] for x in (imgs, ws, [psi])]
            for v in range(c["views"]):
                d.set_view(v, h[0][v], h[1][v], psfs[v])
            d.prepare()
            s.update(decon=d, imgs=h[0], ws=h[1], psi=h[2][0])
        d.synchronize()
    elif c["kind"] in ("block", "block_host"):
        k1, k2, img, w, psi = _block_inputs(c, seed)
        wk = M.BlockWorker((c["x"], c["y"], c["z"]), 1e-4, c["lambda"], 1,
                           M.BOUNDARY_REFERENCE if c["boundary"] == "reference" else M.BOUNDARY_CIRCULAR)
        wk.set_kernels(0, k1, k2)
        if c["kind"] == "block_host":
            img, w, psi = (a.cpu().numpy() for a in (img, w, psi))
        torch.cuda.synchronize()
        s.update(worker=wk, img=img, w=w, psi=psi)
    elif c["kind"] == "fuse":
        views, box = _fuse_inputs(c, seed)
        for v in views:
            v["img_ptr"] = v["img"].data_ptr()
        shape = box[::-1]
        torch.cuda.synchronize()
        s.update(views=views, box=box, image=torch.empty(shape, device=DEV), weight=torch.empty(shape, device=DEV))
    else:
        psi, nxt, tgt = _net_inputs(c, seed)
        net = M.UNet(c["batch"], (c["x"], c["y"], c["z"]), seed=3)
        torch.cuda.synchronize()
        s.update(net=net, psi=psi, next=nxt, target=tgt, pred=torch.empty_like(psi))
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "volume":
        d, out = state["decon"], state["out"]
        d.run_iterations(c["iterations"])
        d.get_psi_device(out.data_ptr())
        return out
    if kind == "host":
        # a time series on the same arrays: the next call's views upload during this one
        return state["decon"].run_host(c["iterations"], state["imgs"], state["ws"], state["psi"], state["imgs"],
                                       state["ws"])
    if kind == "block":
        state["worker"].run_iteration_device(0, state["psi"].data_ptr(), state["img"].data_ptr(), state["w"].data_ptr(),
                                             300.0)
        return state["psi"]
    if kind == "block_host":
        st = state["worker"].run_iteration(0, state["psi"], state["img"], state["w"], 300.0)
        return {"psi": state["psi"], "sum": st.sum_change, "max": st.max_change}
    if kind == "fuse":
        M.fuse_group(state["views"], (0, 0, 0), state["box"], state["image"].data_ptr(), state["weight"].data_ptr())
        return {"image": state["image"], "weight": state["weight"]}
    net = state["net"]
    if kind == "unet_train":
        net.set_input(state["psi"].data_ptr(), state["next"].data_ptr(), state["target"].data_ptr())
        loss = net.train_step(1e-4)
        return {"loss": loss, "grads": net.grads()}
    net.set_input(state["psi"].data_ptr(), state["next"].data_ptr())
    net.forward(state["pred"].data_ptr())
    return state["pred"]


# ---- the work of one pass -----------------------------------------------------------------

def _conv_flops(n):
    """Two FFT convolutions of n real voxels: four real transforms and two spectral products."""
    return 10.0 * n * math.log2(max(2, n)) + 6.0 * n


def work(case):
    c = case
    if c["kind"] in ("unet_train", "unet_forward"):
        n = c["batch"] * c["x"] * c["y"] * c["z"]
        per = [1, 1 / 8, 1 / 64, 1 / 8, 1]  # voxels of each layer's grid
        fl = sum(2.0 * 27 * ci * co * p * n for (ci, co), p in zip(LAYERS, per))
        if c["kind"] == "unet_forward":
            return {"bytes": 12.0 * n, "flops": fl}
        params = sum(27 * ci * co + co for ci, co in LAYERS) + 17
        return {"bytes": 12.0 * n + 4.0 * params * 8, "flops": 3.0 * fl}
    n = c["x"] * c["y"] * c["z"]
    if c["kind"] == "fuse":
        return {"bytes": 4.0 * n * (c["views"] / c["scale_z"] + 2), "flops": 60.0 * n * c["views"]}
    if c["kind"] in ("block", "block_host"):
        return {"bytes": 16.0 * n, "flops": _conv_flops(n) + 10.0 * n}
    item = 4.0 * n
    return {"bytes": item * (2 * c["views"] + 2),
            "flops": c["iterations"] * c["views"] * (_conv_flops(n) + 10.0 * n)}


# ---- the same in 64 bits ------------------------------------------------------------------

def _same(vol, k):
    """Linear convolution with zero extension, output over vol."""
    r = [s // 2 for s in k.shape]
    return _conv(torch.nn.functional.pad(vol, (r[2], r[2], r[1], r[1], r[0], r[0])), k, torch.float64)


def _kernels(c, psfs):
    ks = [torch.from_numpy(p).to(DEV).double() for p in psfs]
    ks = [k / k.sum() for k in ks]

    def flip(k):
        return k.flip(0, 1, 2)

    out = []
    for v, k in enumerate(ks):
        if len(ks) == 1 or c["psf_type"] == "independent":
            out.append((k, flip(k)))
        elif c["psf_type"] == "efficient":
            t = flip(k)
            for w, q in enumerate(ks):
                if w != v:
                    t = t * _same(_same(flip(k), q), flip(q))
            out.append((k, t / t.sum()))
        else:
            t = k
            for w, q in enumerate(ks):
                if w != v:
                    t = t * _same(k, flip(q))
            out.append((k, flip(t / t.sum())))
    return out


def _update(psi, conv2, w, lam, top):
    value = psi * conv2
    if lam > 0:
        v = value.clamp(min=0) / top
        adj = ((1 + 2 * lam * v).sqrt() - 1) / lam * top
    else:
        adj = value
    nxt = torch.where(value > 0, adj, torch.full_like(value, 1e-4)).clamp(min=1e-4)
    return psi + (nxt - psi) * w


def _two_convs(psi, img, k1, k2):
    """conv2 of the quotient: psi extended mirror-single, the quotient by 1."""
    r = [s // 2 for s in k1.shape]
    c1 = _conv(_mirror(psi, r), k1, torch.float64)
    q = torch.where(img > 0, img / c1, torch.ones_like(c1))
    del c1
    return _conv(torch.nn.functional.pad(q, (r[2], r[2], r[1], r[1], r[0], r[0]), value=1.0), k2, torch.float64)


def _exact_volume(c, seed):
    imgs, ws, psfs, psi = _views(c, seed)
    ks = _kernels(c, psfs)
    psi = psi.double()
    tops = [float(i.max()) for i in imgs]
    if c["weights"] == "ones":
        ws = [w.double() for w in ws]
    else:
        # the reference's rule: every weight at most 1, and the sum over the views at most 1
        m = [w.double().clamp(max=1.0) for w in ws]
        total = sum(m)
        ws = [torch.where(total > 1, a / total, a) for a in m]
    for _ in range(c["iterations"]):
        if c["mul"]:
            prod = torch.ones_like(psi)
            for img, (k1, k2) in zip(imgs, ks):
                prod = prod * _two_convs(psi, img.double(), k1, k2)
            root = prod ** (1.0 / c["views"])
            psi = _update(psi, root, sum(ws).clamp(max=1.0), c["lambda"], sum(tops) / len(tops))
        else:
            for img, w, (k1, k2), top in zip(imgs, ws, ks, tops):
                psi = _update(psi, _two_convs(psi, img.double(), k1, k2), w, c["lambda"], top)
    return psi


def _exact_block(c, seed):
    k1, k2, img, w, psi = _block_inputs(c, seed)
    k1, k2 = torch.from_numpy(k1).to(DEV).double(), torch.from_numpy(k2).to(DEV).double()
    old, img = psi.double(), img.double()
    if c["boundary"] == "reference":
        conv2 = _two_convs(old, img, k1, k2)
    else:  # periodic in the block
        def circ(a, k):
            z = torch.zeros_like(a)
            z[:k.shape[0], :k.shape[1], :k.shape[2]] = k
            z = z.roll([-(s // 2) for s in k.shape], (0, 1, 2))
            return torch.fft.irfftn(torch.fft.rfftn(a) * torch.fft.rfftn(z), s=a.shape)

        c1 = circ(old, k1)
        conv2 = circ(torch.where(img > 0, img / c1, torch.ones_like(c1)), k2)
    new = _update(old, conv2, w.double(), c["lambda"], 300.0)
    if c["kind"] == "block":
        return new
    return {"psi": new, "sum": float((new - old).sum()), "max": float((new - old).max())}


def _blend(t, dims, border, rng):
    out = torch.ones(t[0].shape, dtype=torch.float64, device=DEV)
    for d in range(3):
        e = torch.minimum(t[d] - border[d], dims[d] - 1 - t[d] - border[d])
        # the reference's table of the cosine in steps of 1 / 1000
        step = torch.floor((e / rng[d]).clamp(0, 1) * 1000 + 0.5) / 1000
        out = out * torch.where(e <= 0, 0.0, (torch.cos((1 - step) * math.pi) + 1) / 2)
    return out


def _exact_fuse(c, seed):
    views, box = _fuse_inputs(c, seed)
    ax = [torch.arange(n, dtype=torch.float64, device=DEV) for n in box]
    shape = box[::-1]
    si, sw, sd = (torch.zeros(shape, dtype=torch.float64, device=DEV) for _ in range(3))
    for v in views:
        inv = np.linalg.inv(np.vstack([v["model"], [0, 0, 0, 1]]))
        t = [inv[r, 0] * ax[0].view(1, 1, -1) + inv[r, 1] * ax[1].view(1, -1, 1) + inv[r, 2] * ax[2].view(-1, 1, 1) + inv[r, 3]
             for r in range(3)]
        one = torch.ones(shape, dtype=torch.float64, device=DEV)
        wf = _blend(t, v["dims"], *v["fusion"]) if "fusion" in v else one
        wd = _blend(t, v["dims"], *v["decon"]) if "decon" in v else one
        inside = one > 0
        for d in range(3):
            inside = inside & (t[d] > 0) & (t[d] < v["dims"][d] - 1)
        lo = [t[d].floor().clamp(0, v["dims"][d] - 2) for d in range(3)]
        fr = [t[d] - lo[d] for d in range(3)]
        acc = torch.zeros_like(one)
        flat, dx, dxy = v["img"].view(-1), v["dims"][0], v["dims"][0] * v["dims"][1]
        base = (lo[2] * dxy + lo[1] * dx + lo[0]).long()
        for k in range(8):
            o = (k & 1, (k >> 1) & 1, k >> 2)
            q = torch.ones_like(one)
            for d in range(3):
                q = q * (fr[d] if o[d] else 1 - fr[d])
            acc += q * flat[base + o[2] * dxy + o[1] * dx + o[0]].double()
        val = torch.where(inside, acc.clamp(min=1.0), 0.0)
        si += val * wf
        sw += wf
        sd += wd
    return {"image": torch.where(sw > 0, si / sw, 0.0), "weight": sd}


def _exact_net(c, seed):
    """The network in 64 bits without the BF16 rounding of its weights and activations."""
    psi, nxt, tgt = (a.double() for a in _net_inputs(c, seed))
    net = M.UNet(1, (4, 4, 4), seed=3)  # the initial parameters, which are an input
    p = torch.from_numpy(net.params()).to(DEV).double().requires_grad_(c["kind"] == "unet_train")
    net.close()
    F = torch.nn.functional
    o, lay = 0, []
    for ci, co in LAYERS:
        w = p[o:o + co * 27 * ci].view(co, 3, 3, 3, ci).permute(0, 4, 1, 2, 3)
        o += co * 27 * ci
        lay.append((w, p[o:o + co]))
        o += co

    def conv(x, k):
        return F.relu(F.conv3d(x, lay[k][0], lay[k][1], padding=1))

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    x = torch.zeros((c["batch"], 16) + psi.shape[1:], dtype=torch.float64, device=DEV)
    x[:, 0] = torch.log(psi / psi.mean(dim=(1, 2, 3), keepdim=True))
    x[:, 1] = torch.log(nxt / psi)
    e1 = conv(x, 0)
    e2 = conv(F.avg_pool3d(e1, 2), 1)
    b3 = conv(F.avg_pool3d(e2, 2), 2)
    d2 = conv(torch.cat([up(b3), e2], 1), 3)
    d1 = conv(torch.cat([up(d2), e1], 1), 4)
    out = torch.einsum("bczyx,c->bzyx", d1, p[o:o + 16]) + p[o + 16]
    if c["kind"] == "unet_forward":
        return out
    loss = ((out - torch.log(tgt / psi)) ** 2).mean()
    loss.backward()
    return {"loss": float(loss), "grads": p.grad.cpu().numpy()}


def exact(case, seed):
    c = case
    if c["kind"] in ("volume", "host"):
        return _exact_volume(c, seed)
    if c["kind"] in ("block", "block_host"):
        return _exact_block(c, seed)
    if c["kind"] == "fuse":
        return _exact_fuse(c, seed)
    with torch.enable_grad():
        return _exact_net(c, seed)
