"""The PLAIN march's divisions and roots on the device (march_common.cuh: rcp_near,
sqrt_near, div_near, div_by) against CUDA's own IEEE ones: every reciprocal
mantissa, every root mantissa at both exponent parities, and 2^27 quotients over
each of the march's ranges.  The last step corrects by an exact residual, so a
result is off only within 2^-22 of a unit from the middle of two floats, which
for reciprocals and roots of 24-bit numbers leaves none and for quotients at most
a few: the bar is none, and one in 10^7."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

from pedalsky_b200 import build

from . import _gpu

pytestmark = pytest.mark.gpu

RECIPROCAL, ROOT, QUOTIENT, BY_KNOWN, ESTIMATE = range(5)
# numerator and divisor ranges
RANGES = {
    "unit": (1.0, 2.0, 1.0, 2.0),
    "remap": (-1.0, 1.0, 1e-5, 1.0),
    "extinction": (0.0, 1e5, 1e-6, 0.2),
    "altitude": (-1e11, 1e11, 1.2e7, 1.3e7),
    "radius": (-6.46e6, 6.46e6, 6.36e6, 6.46e6),
    "path": (0.0, 1.2e6, 1.0, 1.2e6),
    "scale": (-4e5, 4e5, 1.0, 5e4),
    "thickness": (0.0, 1.2e4, 1.0, 1.2e4),
}


@pytest.fixture(scope="module")
def count(tmp_path_factory):
    _gpu.torch_cuda()
    so = tmp_path_factory.mktemp("near") / "near_division.so"
    here = Path(__file__).resolve().parent
    subprocess.run([build._nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I", str(build.ROOT / "include"), "-I", str(build.CSRC), str(here / "near_division.cu"),
                    "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.count_off.argtypes = [C.c_int] + [C.c_float] * 4 + [C.c_uint64, C.POINTER(C.c_uint64)]

    def run(what, x0, x1, y0, y1, n):
        off = C.c_uint64(0)
        assert lib.count_off(what, x0, x1, y0, y1, n, C.byref(off)) == 0
        return off.value
    return run


def test_every_reciprocal_and_root(count):
    for exponent in (-100, -20, 0, 23, 100):
        assert count(RECIPROCAL, 2.0 ** exponent, 0, 0, 0, 1 << 23) == 0, exponent
        assert count(ROOT, 2.0 ** exponent, 0, 0, 0, 1 << 24) == 0, exponent


@pytest.mark.parametrize("name", sorted(RANGES))
def test_quotients(count, name):
    n = 1 << 27
    assert count(ESTIMATE, *RANGES[name], n) > n // 50  # the uncorrected estimate is off often
    for what in (QUOTIENT, BY_KNOWN):
        assert count(what, *RANGES[name], n) <= n // 10_000_000, (name, what)
