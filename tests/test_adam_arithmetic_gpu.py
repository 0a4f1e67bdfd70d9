"""The straight-line division, reciprocal and square root of Adam give the bits of CUDA's correctly rounded
ones over the ranges in which AdamOp::vec uses them."""
import ctypes as C
import os
import subprocess

import pytest

from raf_b200 import build

pytestmark = pytest.mark.gpu


class Found(C.Structure):
    _fields_ = [("count", C.c_ulonglong), ("a", C.c_float), ("b", C.c_float)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("native") / "arithmetic.so")
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "native_adam_arithmetic.cu")
    subprocess.run([build._nvcc()] + build.NVCC_FLAGS + ["-shared", "-o", out, src], check=True)
    lib = C.CDLL(out)
    lib.check_quotients.argtypes = [C.c_int] * 4 + [C.c_longlong, C.c_void_p]
    return lib


def none(call, *args):
    found = Found()
    assert call(*args, C.byref(found)) == 0
    assert found.count == 0, (found.count, float(found.a).hex(), float(found.b).hex())


# denominators are sqrt(v / bc2) + eps: 2^-50 or eps (2^-40 at least) to 2^31
def test_reciprocal(lib):
    none(lib.check_significands, 0, -60, 60)


# v / bc2 with v of 2^-100 .. 2^40, bc2 of 2^-20 .. 1
def test_square_root(lib):
    none(lib.check_significands, 1, -100, 100)


@pytest.mark.parametrize("a,b", [((-80, 59), (-20, -1)),  # m / bc1
                                 ((-100, 39), (-20, -1)),  # v / bc2
                                 ((-80, 79), (-40, 31)),  # (m / bc1) / denominator
                                 ((-80, -80), (-20, -20)), ((-80, -79), (30, 31)), ((78, 79), (-40, -40))])  # the corners
def test_division(lib, a, b):
    none(lib.check_quotients, *a, *b, 1 << 28)
