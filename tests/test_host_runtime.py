"""The library's host code on a stand-in for the CUDA runtime (fake_cudart.c): devices that the calling
thread is not on, and calls that fail.  No kernel runs; what is checked is which device memory is
allocated on, whether launches are accepted, and that a call after a failed one starts over."""
import os
import subprocess
import sys

import pytest

import build_lib

HERE = os.path.dirname(os.path.abspath(__file__))
PRELUDE = """
import ctypes as C, numpy as np, sys
sys.path[:0] = [{pkg!r}]
import mvrgb300 as M
F = C.CDLL({fake!r})
F.fake_live.restype = F.fake_launches.restype = C.c_longlong
F.fake_fail.argtypes = [C.c_int, C.c_longlong]
MALLOC, LAUNCH = 0, 1
K = lambda n: np.ones(n[::-1], np.float32) / np.prod(n)
A = lambda b, n=None: np.ones(b[::-1], np.float32) if n is None else [np.ones(b[::-1], np.float32) for _ in range(n)]
"""


@pytest.fixture(scope="session")
def fake(tmp_path_factory):
    build_lib.build()
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(build_lib._nvcc())), "include")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", f"-I{inc}", "-o", so, os.path.join(HERE, "fake_cudart.c")], check=True)
    return so


def run(fake, body, devices=2, **env):
    pre = PRELUDE.format(pkg=build_lib.HERE, fake=fake)
    e = {k: v for k, v in os.environ.items() if not k.startswith("MVR_")}
    r = subprocess.run([sys.executable, "-c", pre + body], capture_output=True, text=True, timeout=120,
                       env=dict(e, LD_PRELOAD=fake, FAKE_DEVICES=str(devices), **env))
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout


# a Mul block with one view off the separable transforms: its plan and the other view's are block plans
MIXED = """
b = (40, 8, 24)
def make():
    w = M.BlockWorker(b, num_views=2, device=1)
    for v, k in enumerate(((5, 5, 5), (5, 21, 5))):
        w.set_kernels(v, K(k), K(k))
    return w
def step(w):
    n = F.fake_launches()
    w.run_iteration_mul(A(b), A(b, 2), A(b, 2), [1.0, 1.0])
    return F.fake_launches() - n
"""


def test_mixed_mul_block_on_another_device_than_the_threads(fake):
    run(fake, MIXED + """
w = make()
assert F.cudaSetDevice(0) == 0
n0 = F.fake_live(0)
step(w)
assert F.fake_live(0) == n0, "memory of device 0"
""")


@pytest.mark.parametrize("kind", ["MALLOC", "LAUNCH"])
def test_mixed_mul_block_after_a_plan_that_failed(fake, kind):
    # whichever allocation (three tables, two spectra; then the step's own) or launch of the plan fails,
    # the next call makes it anew
    run(fake, MIXED + f"""
w = make()
first, later = step(w), step(w)
assert first > later  # the first made the plan
failed = 0
for i in range(12 if {kind} == MALLOC else first - later):
    w = make()
    F.fake_fail({kind}, i)
    try:
        step(w)
        F.fake_fail({kind}, -1)
        continue  # fewer allocations than that
    except M.MvrError:
        failed += 1
    assert (step(w), step(w)) == (later if {kind} == MALLOC and i >= 5 else first, later), i
assert failed >= 4
""")


# kernels with more than 48 KB of shared memory: y and z lengths from 360 and x length 576 of the separable
# transforms, the plane and pair kernels, the row / column kernels
@pytest.mark.parametrize("block,env", [
    ((572, 356, 476), {}), ((316, 60, 356), {}), ((188, 188, 60), {"MVR_PLANE_KERNELS": "1"}),
    ((252, 252, 60), {"MVR_PAIR_KERNELS": "1"}), ((236, 500, 404), {"MVR_PLANE_KERNELS": "0"}),
])
def test_every_device_gets_the_shared_memory_of_the_kernels(fake, block, env):
    run(fake, f"""
b = {block}
for dev in (0, 1):
    w = M.BlockWorker(b, device=dev)
    w.set_kernels(0, K((5, 5, 5)), K((5, 5, 5)))
    w.run_iteration(0, A(b), A(b), A(b), 1.0)
""", **env)


def test_block_without_room_for_the_separable_transforms(fake):
    # each of the first allocations fails in turn: the block's kernels are taken all the same (a block plan,
    # whose domain is the smaller one), with the bytes that a block plan alone would hold
    run(fake, """
import os
b, k = (33, 33, 33), (5, 5, 5)
def live(fail):
    w = M.BlockWorker(b, device=1)
    n0 = F.fake_live(1)
    F.fake_fail(MALLOC, fail)
    w.set_kernels(0, K(k), K(k))
    F.fake_fail(MALLOC, -1)
    n1 = F.fake_live(1) - n0
    w.run_iteration(0, A(b), A(b), A(b), 1.0)
    return n1
sep = live(-1)
os.environ["MVR_RATIO_BAND"] = "0"
plan = live(-1)
del os.environ["MVR_RATIO_BAND"]
assert plan < sep
assert [live(i) for i in (0, 2, 3, 4, 6, 7, 8)] == [plan] * 7
""")


def test_volume_without_room_for_the_tiles(fake):
    # as above for the tiles of a volume: prepare succeeds, the step stays on its blocks
    run(fake, """
D, b, k = (40, 36, 24), (48, 40, 32), (5, 5, 5)
def prepare(fail, n):
    with M.Deconvolution(D, n, b, psf_type=M.PSF_INDEPENDENT, filter_blocks=False, device=1) as d:
        for v in range(n):
            d.set_view(v, A(D), A(D), K(k))
        F.fake_fail(MALLOC, fail)
        try:
            d.prepare()
        except M.MvrError:
            return None
        finally:
            F.fake_fail(MALLOC, -1)
        n0 = F.fake_launches()
        d.run_iterations(1)
        return F.fake_launches() - n0
tiles, n = prepare(-1, 1), 0
while prepare(n, 1) is None:  # allocations of the block plans
    n += 1
rest = [prepare(i, 1) for i in range(n, n + 10)]  # two for the blocks' levels, three tables, two spectra, marks
assert len(set(rest[:8])) == 1 and rest[0] not in (None, tiles) and rest[8:] == [tiles] * 2, (tiles, n, rest)
""")


@pytest.mark.parametrize("dims,block,views,mul,fp64", [
    ((40, 36, 24), (48, 40, 32), 2, False, False), ((40, 36, 24), (48, 40, 32), 3, True, False),
    ((40, 36, 24), (48, 40, 32), 2, False, True), ((40, 36, 24), (48, 40, 32), 2, True, True),
    ((280, 280, 280), (300, 300, 300), 2, False, False), ((280, 280, 280), (300, 300, 300), 3, True, False),  # slabs
    ((1180, 40, 36), (120, 60, 60), 2, True, True),  # several FP64 tiles
])
def test_launch_count(fake, dims, block, views, mul, fp64):
    # what the handle reports is what the runtime was asked for
    run(fake, f"""
D, b, n = {dims}, {block}, {views}
with M.Deconvolution(D, n, b, mul={mul}, psf_type=M.PSF_INDEPENDENT, filter_blocks=False,
                     precision=M.PRECISION_FP64 if {fp64} else M.PRECISION_FP32) as d:
    for v in range(n):
        d.set_view(v, A(D), A(D), K((5, 5, 5)))
    d.prepare()
    d.set_graphs(False)
    for _ in range(2):
        f0, c0 = F.fake_launches(), d.launch_count()
        d.run_iterations(1)
        assert F.fake_launches() - f0 == d.launch_count() - c0, (F.fake_launches() - f0, d.launch_count() - c0)
""")


def test_more_blocks_than_a_grid_has_rows(fake):
    # 70000 blocks of 16 voxels, 12 apart: prepare looks at their levels in one launch
    run(fake, """
D = (840000, 3, 3)
with M.Deconvolution(D, 1, (16, 16, 16), psf_type=M.PSF_INDEPENDENT, filter_blocks=False) as d:
    d.set_view(0, A(D), A(D), K((3, 3, 3)))
    d.prepare()
    d.run_iterations(1)
""")
