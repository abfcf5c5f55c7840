"""The straight-line reciprocal, square root and quotient (csrc/sx_exact.cuh) against
the compiler's correctly rounded ones: the first two over every float32 of their
range, the quotient over every numerator that its error bound leaves open."""
import ctypes as C
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "starlab-physics_gb300", "csrc")


@pytest.fixture(scope="module")
def check(pkg, tmp_path_factory):
    from starlab_physics_gb300 import build

    so = str(tmp_path_factory.mktemp("exact") / "exact_check.so")
    subprocess.run([build.nvcc_path(), *build.NVCC_FLAGS, "-I" + CSRC, "-shared", "-o", so,
                    os.path.join(HERE, "native", "exact_check.cu")], check=True)
    lib = C.CDLL(so)
    lib.check.argtypes = [C.c_int, C.c_uint, C.c_uint, C.c_int, C.c_int, C.c_int, C.POINTER(C.c_ulonglong * 2)]

    def run(what, first=0, last=0, reach=0, ea=0, eb=0):
        out = (C.c_ulonglong * 2)()
        assert lib.check(what, first, last, reach, ea, eb, C.byref(out)) == 0
        return out[0], out[1]

    return run


def _bits(exponent):
    return (127 + exponent) << 23


def test_reciprocal(check):
    """2^-100 <= |x| < 2^126 (SiLU divides by up to 2^126)."""
    assert check(0, _bits(-100), _bits(126)) == (0, 2 * 226 << 23)


def test_square_root(check):
    assert check(1, _bits(-100), _bits(100) + 1) == (0, (200 << 23) + 1)


@pytest.mark.parametrize("ea,eb", [(0, 0), (0, 1), (-100, 0), (100, 99), (-60, 60), (20, -100), (6, 125)])
def test_quotient_next_to_midpoints(check, ea, eb):
    bad, done = check(2, reach=8, ea=ea, eb=eb)
    assert bad == 0 and done > 10_000_000
