"""The FP32 estimate that lets rain_ice skip an IEEE division: quot_above may
say "above" only where the exact quotient is above the bound, over bounds from
far below FP32's normal range to far above it, zero, infinite and NaN; and it
does say so for a quotient that is 2^-16 above an ordinary bound."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def above(tmp_path_factory):
    out = tmp_path_factory.mktemp("est") / "libest_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(HERE, "..", "include"), os.path.join(HERE, "estimate_host.cpp"), "-o", str(out)],
                   check=True)
    lib = ctypes.CDLL(str(out))

    def run(num, den, bound):
        a = [np.ascontiguousarray(v, dtype=np.float64) for v in np.broadcast_arrays(num, den, bound)]
        r = np.empty(a[0].size, dtype=np.int32)
        lib.quot_above_host(ctypes.c_long(r.size), *[v.ctypes.data_as(ctypes.c_void_p) for v in a],
                            r.ctypes.data_as(ctypes.c_void_p))
        return r.astype(bool)
    return run


@pytest.mark.parametrize("lo,hi", [(-140, -120), (-1070, -126), (-127, -125), (-30, 30), (120, 140), (126, 1000)])
def test_above_is_certain(above, lo, hi):
    rng = np.random.default_rng(abs(lo))
    n = 4000
    den = 2.0 ** rng.uniform(-100, 100, n) * rng.choice([-1.0, 1.0], n)
    bound = 2.0 ** rng.uniform(lo, hi, n) * rng.choice([-1.0, 1.0], n, p=[0.25, 0.75])
    near = np.clip(np.abs(bound) * 2.0 ** rng.uniform(-3, 3, n), 2.0 ** -225, 2.0 ** 225)   # quotients around the bound
    num = near * den * rng.choice([-1.0, 1.0], n, p=[0.25, 0.75])
    for i in np.flatnonzero(above(num, den, bound)):
        assert Fraction(num[i]) / Fraction(den[i]) > Fraction(bound[i])


def test_special_bounds(above):
    assert not above(1.0, 3.0, [np.inf, np.nan, -np.nan]).any()
    assert not above(-1.0, 3.0, [0.0, -0.0]).any()
    assert not above([0.0, np.nan, np.inf, 1.0, 1.0], [1.0, 1.0, 1.0, 0.0, np.nan], 0.0).any()


def test_ordinary_quotients_are_seen(above):
    rng = np.random.default_rng(9)
    bound, den = 2.0 ** rng.uniform(-60, 60, 2000), 2.0 ** rng.uniform(-30, 30, 2000)
    assert above(bound * (1 + 2.0 ** -16) * den, den, bound).all()
