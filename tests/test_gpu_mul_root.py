"""The root of the Mul update's running product for every number of views: a float rounding of the exact
root, 2^-24, and 1 % of that for the sum that is rounded."""
import ctypes as C
import os
import subprocess

import pytest

import build_lib

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("root") / "libroot.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "mul_root_check.cu")
    subprocess.run([build_lib._nvcc(), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared",
                    "-Xcompiler", "-fPIC", f"-I{build_lib.CSRC}", "-o", so, src], check=True)
    lib = C.CDLL(so)
    lib.root_error.restype = C.c_double
    return lib


@pytest.mark.parametrize("views", range(2, 17))
def test_root_is_rounded_once(lib, views):
    assert 0 <= lib.root_error(views, 1 << 20) <= 1.01 * 2.0 ** -24
