"""The fixed-point exp / exp10 / log / atan of fastmath.cuh (host build of the
kernels' source) where they can go wrong: at the edges of the reduction and of
the table intervals, next to x = 1, in the last normal binades and across the
gradual underflow, against 200-bit mpmath values.  The fixed-point error is
below 2^-58 of the result, so the rounded results are within 0.55 ulp (1 ulp
where the result is subnormal or an FP64 form is used: log next to x = 1, atan
below 2^-7)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

mp = pytest.importorskip("mpmath")

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def ev(tmp_path_factory):
    out = tmp_path_factory.mktemp("ffp") / "libfm_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(HERE, "fastmath_host.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.fm_eval.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long]

    def run(fn, x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.empty_like(x)
        lib.fm_eval(fn, x.ctypes.data, y.ctypes.data, x.size)
        return y
    return run


def around(x, n=2):
    """Each x and its n neighbours on both sides."""
    x = np.asarray(x, dtype=np.float64)
    lo, hi, out = x, x, [x]
    for _ in range(n):
        lo, hi = np.nextafter(lo, -np.inf), np.nextafter(hi, np.inf)
        out += [lo, hi]
    return np.concatenate(out)


def worst_ulp(got, fn, xs):
    mp.mp.prec = 200
    w = 0.0
    for g, x in zip(got, xs):
        e = fn(mp.mpf(float(x)))
        w = max(w, float(abs(mp.mpf(float(g)) - e) / np.spacing(abs(float(e)))))
    return w


LN2 = float(np.log(2.0))
RNG = np.random.default_rng(11)
CASES = {
    "exp-steps": (0, around(np.arange(-3000, 3000, 7) * (LN2 / 512)), 0.55),
    "exp-large": (0, around(RNG.integers(-360000, 520000, 400) * (LN2 / 512)), 0.55),
    "exp-small": (0, np.concatenate([s * 2.0 ** RNG.uniform(-80, -5, 300) for s in (1, -1)]), 0.55),
    "exp-normal-ends": (0, RNG.uniform([[-708.39], [709.0]], [[-700.0], [709.78]], (2, 200)).ravel(), 0.55),
    "exp-subnormal": (0, RNG.uniform(-744.0, -708.4, 300), 1.0),
    "exp10-steps": (1, around(np.arange(-2000, 2000, 11) * (np.log10(2.0) / 512)), 0.55),
    "exp10-large": (1, RNG.uniform(-307.0, 308.2, 400), 0.55),
    "log-intervals": (2, around(np.outer(1 + np.arange(0, 512, 3) / 512, [0.25, 2.0, 1024.0]).ravel(), 1), 0.55),
    "log-beside-one": (2, around(np.concatenate([1 + 2.0 ** -8 + np.arange(8) * 2.0 ** -12,
                                                 1 - 2.0 ** -8 - np.arange(1, 9) * 2.0 ** -12])), 0.55),
    "log-at-one": (2, np.concatenate([1 + s * 2.0 ** RNG.uniform(-52, -8.001, 300) for s in (1, -1)]), 1.0),
    "log-binades": (2, 2.0 ** RNG.uniform(-1022, 1023.9, 500), 0.55),
    "log-subnormal": (2, 2.0 ** RNG.uniform(-1073, -1022, 200), 0.55),
    "atan-table-steps": (4, around(np.concatenate([np.arange(1, 65) / 64, (np.arange(1, 65) - 0.5) / 64])), 0.55),
    "atan-reciprocal-steps": (4, around(64 / np.concatenate([np.arange(1, 65), np.arange(1, 65) - 0.5])), 0.55),
    "atan-at-one": (4, around([1.0, -1.0], 4), 0.55),
    "atan-small-end": (4, around([2.0 ** -7, -2.0 ** -7], 4), 1.0),
    "atan-range": (4, np.concatenate([s * 2.0 ** RNG.uniform(-6.9, 59.9, 400) for s in (1, -1)]), 0.55),
    "atan-small": (4, np.concatenate([s * 2.0 ** RNG.uniform(-40, -7, 300) for s in (1, -1)]), 1.0),
}


@pytest.mark.parametrize("name", list(CASES))
def test_within_bound(ev, name):
    fn, xs, bound = CASES[name]
    exact = (mp.exp, lambda v: mp.power(10, v), mp.log, None, mp.atan)[fn]
    xs = xs[xs != 1.0] if fn == 2 else xs
    assert worst_ulp(ev(fn, xs), exact, xs) <= bound
