"""Device functions on their own (device_units.cu, compiled here), at the ends of
their ranges: division by a known divisor, the stopping test on the squared
residual, and the dense inverse of the coarsest multigrid level."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import cases
from rans_sst_py import _build

pytestmark = pytest.mark.gpu

_dp, _ip = C.POINTER(C.c_double), C.POINTER(C.c_int32)


def _d(a):
    return a.ctypes.data_as(_dp)


_built = []   # once per process: test_gpu_vcycle.py uses it too


@pytest.fixture(scope="module")
def units(tmp_path_factory):
    if not _built:
        so = str(tmp_path_factory.mktemp("units") / "device_units.so")
        subprocess.run([_build.nvcc()] + _build.ARCH + ["-O3", "-std=c++17", "-fmad=false", "-shared", "-Xcompiler",
                                                        "-fPIC", "-I", _build.INCLUDE, cases.HERE + "/device_units.cu",
                                                        "-o", so, "-cudart", "static"], check=True)
        _built.append(C.CDLL(so))
    return _built[0]


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


def test_stopping_test(units):
    """sq < limit as sqrt(sq) / r0 < tol, for sq a few units around the limit and
    far from it, with the norms and tolerances from one end of the range to the other."""
    rng = np.random.default_rng(2)
    e = np.array([-320, -300, -200, -141, -140, -139, -71, -70, -69, -30, -8, -3, 0, 3, 30, 69, 70, 71, 139, 140, 141, 300])
    with np.errstate(all="ignore"):
        r0 = np.repeat(rng.uniform(1.0, 9.9, len(e)) * np.power(10.0, e), len(e))
        tol = np.tile(rng.uniform(1.0, 9.9, len(e)) * np.power(10.0, e), len(e))
        r0 = np.concatenate([r0, 10.0 ** rng.uniform(-20, 5, 2000), [1.0, 1.0, 1.0, 0.0, np.inf, np.nan, 1.0]])
        tol = np.concatenate([tol, 10.0 ** rng.uniform(-12, 0, 2000), [0.0, -1.0, np.inf, 1.0, 1.0, 1.0, np.nan]])
        at = (r0 * tol) ** 2
        steps = np.concatenate([np.arange(-40, 41), [-10 ** 6, 10 ** 6]])
        near = np.maximum(np.where(np.isfinite(at), at, 1.0).view(np.int64)[:, None] + steps, 0).view(np.float64)
        far = np.array([0.0, 5e-324, 1e-300, 1.0, 1e300, np.inf, np.nan])
        sq = np.concatenate([near, np.broadcast_to(far, (len(r0), len(far)))], 1).copy()
        want = np.sqrt(sq) / r0[:, None] < tol[:, None]
    below, limit = np.empty(sq.shape, np.int32), np.empty(len(r0))
    assert units.unit_residual_limit(len(r0), sq.shape[1], _d(r0), _d(tol), _d(sq), below.ctypes.data_as(_ip),
                                     _d(limit)) == 0
    # a zero start never reaches the test: the solvers end on it
    use = ~(r0 == 0.0)
    assert np.array_equal(below[use] != 0, want[use])
    # ordinary norms and tolerances take the limit, not the division
    assert np.all(np.isfinite(limit[(r0 > 1e-20) & (r0 < 1e6) & (tol > 1e-13) & (tol < 1.0)]))


def _spd(n, rng):
    """Condition number of about 1e3."""
    a = rng.normal(size=(n, n)) / np.sqrt(n)
    a = a @ a.T
    return a + np.eye(n) * (4.0 / 999.0)


def _inverse(units, a, blocks, threads=512):
    x, ok = a.copy(), np.full(max(blocks, 1), -1, np.int32)
    assert units.unit_dense_inverse(blocks, threads, len(a), _d(x), ok.ctypes.data_as(_ip)) == 0
    assert len(set(ok.tolist())) == 1
    return x, ok[0] == 1


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 100, 511, 709, 972, 1024])
def test_dense_inverse(units, n):
    """X A = I to 8 n eps cond; the same bits for any number of CTAs, and in the
    one-CTA form."""
    a = _spd(n, np.random.default_rng(n))
    x, good = _inverse(units, a, 64)
    assert good
    cond = np.linalg.cond(a)
    assert np.abs(x @ a - np.eye(n)).max() <= 8 * n * np.finfo(float).eps * cond
    for blocks in (1, 5, 128):
        if blocks == 1 and n > 512:
            continue
        other, good = _inverse(units, a, blocks)
        assert good and np.array_equal(other, x), blocks
    if n <= 32:
        for threads in (256, 512):
            other, good = _inverse(units, a, 0, threads)
            assert good and np.array_equal(other, x), threads


@pytest.mark.parametrize("n,k", [(1, 0), (16, 15), (17, 16), (32, 7), (50, 0), (50, 31), (50, 49), (300, 160)])
@pytest.mark.parametrize("kind", ["zero", "nan", "tiny"])
def test_vanishing_pivot_is_reported(units, n, k, kind):
    """On every CTA, so that the whole team goes on with the other form."""
    a = np.diag(np.arange(1.0, n + 1.0))
    a[k, k] = dict(zero=0.0, nan=np.nan, tiny=1e-301)[kind]
    for blocks in (1, 40):
        assert not _inverse(units, a, blocks)[1]
    if n <= 32:
        for threads in (256, 512):
            assert not _inverse(units, a, 0, threads)[1]
