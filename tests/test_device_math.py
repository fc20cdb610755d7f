"""The device arithmetic that the field kernels take for exact (GPU): the
reciprocal and quotient without the division's slow path against the division,
the sphere exit of a unit direction against the general one, ex2 near 0, and
the dust update with the fast quotient against the same with the division."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def device_math(tmp_path_factory):
    from portal_gb300 import build
    so = str(tmp_path_factory.mktemp("math") / "device_math.so")
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared",
                    "-I", build.CSRC, "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "device_math.cu"), "-o", so], check=True, capture_output=True)
    f = C.CDLL(so).device_math
    f.argtypes, f.restype = [C.c_int, C.c_longlong], C.c_longlong
    return f


@pytest.mark.parametrize("which,count", [(0, 0), (1, 1 << 32), (2, 3 << 26), (3, 0), (4, 1 << 30)],
                         ids=["reciprocal", "quotient", "sphere_exit", "ex2", "dust"])
def test_no_exceptions(device_math, which, count):
    assert device_math(which, count) == 0
