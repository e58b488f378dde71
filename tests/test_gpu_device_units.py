"""Device functions on their own (device_units.cu, compiled here), at the ends of
their ranges: division by a known divisor."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import cases
from rans_sst_py import _build

pytestmark = pytest.mark.gpu

_dp = C.POINTER(C.c_double)


def _d(a):
    return a.ctypes.data_as(_dp)


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("units") / "device_units.so")
    subprocess.run([_build.nvcc()] + _build.ARCH + ["-O3", "-std=c++17", "-fmad=false", "-shared", "-Xcompiler", "-fPIC",
                                                    "-I", _build.INCLUDE, cases.HERE + "/device_units.cu", "-o", so,
                                                    "-cudart", "static"], check=True)
    return C.CDLL(so)


def _same(a, b):
    """Equal as doubles, the sign of zero included; NaNs are alike."""
    return (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))


def test_division_by_known_divisor(units):
    """x / d bit for bit: exponents all over, at the ends of the ranges that take
    the multiplication, where the quotient leaves the normal numbers, and what is
    no ordinary number."""
    rng = np.random.default_rng(1)
    ends = np.array([-1074, -1022, -1000, -700, -621, -620, -619, -310, -301, -300, -299, -52, -1, 0, 1, 52, 299, 300,
                     301, 310, 619, 620, 621, 700, 1000, 1023])
    ex, ed = np.repeat(ends, len(ends)), np.tile(ends, len(ends))
    ex, ed = np.tile(ex, 400), np.tile(ed, 400)
    wide = rng.integers(-1074, 1024, (2, 200000))
    ex, ed = np.concatenate([ex, wide[0]]), np.concatenate([ed, wide[1]])
    sign = lambda: rng.choice([-1.0, 1.0], len(ex))  # noqa: E731
    with np.errstate(all="ignore"):
        x = np.ldexp(sign() * rng.uniform(1.0, 2.0, len(ex)), ex)
        d = np.ldexp(sign() * rng.uniform(1.0, 2.0, len(ex)), ed)
        odd = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 2.2250738585072014e-308, 1.7976931348623157e308, 1.0])
        x = np.concatenate([x, np.repeat(odd, len(odd)), np.repeat(odd, len(ends))])
        d = np.concatenate([d, np.tile(odd, len(odd)), np.tile(np.ldexp(1.5, ends), len(odd))])
        r, want = 1.0 / d, x / d
    q = np.empty_like(x)
    assert units.unit_div_by(len(x), _d(x), _d(d), _d(r), _d(q)) == 0
    wrong = np.flatnonzero(~_same(q, want))
    assert len(wrong) == 0, [(x[i], d[i], q[i], want[i]) for i in wrong[:5]]
