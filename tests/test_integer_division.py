"""The integer reciprocal and division of fastmath.cuh (host build of the
kernels' source): the IEEE results bit for bit at the edges of their paths -
significands near 1 and 2, quotients next to a power of two, the ends of the
exponent range, zeros, subnormals, infinities and NaN."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("idiv") / "libfm_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(HERE, "fastmath_host.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.fm_eval.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]
    lib.fm_div.argtypes = [ctypes.c_int] + [ctypes.c_void_p] * 4 + [ctypes.c_long]
    return lib


def significands(rng, n):
    """Doubles in [1, 2): near 1, near 2, short and random ones."""
    one = np.float64(1.0).view(np.uint64)
    bits = np.concatenate([np.arange(64), 2 ** 52 - 1 - np.arange(64), rng.integers(0, 64, n) << 46,
                           rng.integers(0, 2 ** 52, n)]).astype(np.uint64)
    return (bits + one).view(np.float64)


@pytest.mark.parametrize("ea,eb", [(0, 0), (-1, 1), (500, -500), (-500, 500), (-1022, 0), (-1022, 1), (1023, 0),
                                   (1023, -1), (0, 1023), (0, 1022), (0, -1022), (511, -511), (512, -511),
                                   (-511, 510), (-511, 511), (-511, 512)])
def test_division_is_ieee(lib, ea, eb):
    rng = np.random.default_rng(abs(ea) * 7 + abs(eb))
    m = significands(rng, 2000)
    a = np.ldexp(rng.permutation(m), ea) * rng.choice([-1.0, 1.0], m.size)
    b = np.ldexp(rng.permutation(m), eb) * rng.choice([-1.0, 1.0], m.size)
    a = np.concatenate([a, a, np.where(np.abs(b) < 1e300, b, b / 4.0) * 3.0])
    b = np.concatenate([b, a[: b.size], b])
    sp = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2e-308, 1.7976931348623157e308, 1.0])
    a = np.concatenate([a, np.repeat(sp, sp.size)])
    b = np.concatenate([b, np.tile(sp, sp.size)])
    q, q2, r = np.empty_like(a), np.empty_like(a), np.empty_like(a)
    with np.errstate(all="ignore"):
        for mode in (0, 1):
            lib.fm_div(mode, a.ctypes.data, b.ctypes.data, q.ctypes.data, q2.ctypes.data, a.size)
            want = a / b
            ok = np.isnan(want)
            assert np.array_equal(np.isnan(q), ok)
            assert np.array_equal(q[~ok].view(np.uint64), want[~ok].view(np.uint64))
        want2 = (2.5 * a) / b
        ok = np.isnan(want2)
        assert np.array_equal(q2[~ok].view(np.uint64), want2[~ok].view(np.uint64))
        lib.fm_eval(3, b.ctypes.data, r.ctypes.data, b.size)
        want = 1.0 / b
        ok = np.isnan(want)
        assert np.array_equal(np.isnan(r), ok) and np.array_equal(r[~ok].view(np.uint64), want[~ok].view(np.uint64))
