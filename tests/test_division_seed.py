"""The integer reciprocal and division with a seed one and two units of the
last place below and above the rounded FP32 reciprocal: the device's
approximation may be one unit off the exact value, which for a divisor next to
2 reaches two below the rounded one, the value below 1/2.  The IEEE results all
the same; and the arc tangent, which uses the same reciprocal, within its
0.55 ulp."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_integer_division import significands

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", params=[-2, -1, 1, 2])
def lib(request, tmp_path_factory):
    out = tmp_path_factory.mktemp("seed") / "libfm_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    f"-DFM_HOST_SEED_ULPS={request.param}", os.path.join(HERE, "fastmath_host.cpp"), "-o", str(out)],
                   check=True)
    lib = ctypes.CDLL(str(out))
    lib.fm_eval.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]
    lib.fm_div.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 4 + [ctypes.c_long]
    return lib


def _divisors():
    """Every FP32 significand of the last 64 below 2 and the first 64 from 1,
    with the low bits at both ends and random, and the general ones."""
    rng = np.random.default_rng(2)
    top = np.concatenate([2 ** 23 - 1 - np.arange(64), np.arange(64)]).astype(np.uint64) << np.uint64(29)
    low = np.concatenate([np.array([0, 1, 2 ** 29 - 1]), rng.integers(0, 2 ** 29, 13)]).astype(np.uint64)
    near = ((top[:, None] | low[None, :]).ravel() + np.float64(1.0).view(np.uint64)).view(np.float64)
    return np.concatenate([near, significands(rng, 3000)])


def test_reciprocal_and_quotient_are_ieee(lib):
    b = _divisors()
    a = np.random.default_rng(3).permutation(b)
    r, q, q2 = np.empty_like(b), np.empty_like(b), np.empty_like(b)
    lib.fm_eval(3, b.ctypes.data, r.ctypes.data, b.size)
    assert np.array_equal(r, 1.0 / b)
    lib.fm_div(0, a.ctypes.data, b.ctypes.data, q.ctypes.data, q2.ctypes.data, b.size)
    assert np.array_equal(q, a / b)
    lib.fm_div(1, a.ctypes.data, b.ctypes.data, q.ctypes.data, q2.ctypes.data, b.size)
    assert np.array_equal(q, a / b) and np.array_equal(q2, (2.5 * a) / b)


def test_arc_tangent(lib):
    mp = pytest.importorskip("mpmath")
    mp.mp.prec = 200
    x = np.concatenate([_divisors()[::7], 1.0 / _divisors()[::7], 2.0 ** np.random.default_rng(5).uniform(-6.9, 20, 300)])
    y = np.empty_like(x)
    lib.fm_eval(4, x.ctypes.data, y.ctypes.data, x.size)
    for v, g in zip(x, y):
        e = mp.atan(mp.mpf(float(v)))
        assert abs(mp.mpf(float(g)) - e) <= 0.55 * float(np.spacing(float(e)))
