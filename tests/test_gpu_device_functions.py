"""The device build of fastmath.cuh against its host build, on the arguments
of the host tests.  exp, exp10, log, the reciprocal, the divisions and the
square roots are exact integer and explicitly rounded operations from seeds
that cannot reach the result, so they agree bit for bit (a NaN counts as
equal to a NaN).  The arc tangent does not settle its quotient: the device's
approximate seed may move its last bit.  The seed itself is within one unit
of the last place of the rounded reciprocal for every significand."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from test_fixed_point_functions import CASES
from test_integer_division import significands

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2e-308, 1.7976931348623157e308, 1.0, -1.0])


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    sys.path.insert(0, os.path.join(HERE, "..", "dwarf-p-ice3_gb300"))
    import build
    d = tmp_path_factory.mktemp("fm")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    os.path.join(HERE, "fastmath_device.cu"), "-o", str(d / "libfm_device.so")], check=True)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    os.path.join(HERE, "fastmath_host.cpp"), "-o", str(d / "libfm_host.so")], check=True)
    return ctypes.CDLL(str(d / "libfm_device.so")), ctypes.CDLL(str(d / "libfm_host.so"))


def device(libs, fn, a, b=None):
    ta = torch.as_tensor(np.ascontiguousarray(a)).cuda()
    tb = ta if b is None else torch.as_tensor(np.ascontiguousarray(b)).cuda()
    q, q2 = torch.empty_like(ta), torch.empty_like(ta)
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in (ta, tb, q, q2)]
    assert libs[0].fm_eval_device(fn, *p, ctypes.c_long(ta.numel())) == 0
    return q.cpu().numpy(), q2.cpu().numpy()


def host(libs, fn, a):
    a = np.ascontiguousarray(a)
    y = np.empty_like(a)
    libs[1].fm_eval(fn, ctypes.c_void_p(a.ctypes.data), ctypes.c_void_p(y.ctypes.data), ctypes.c_long(a.size))
    return y


def same(a, b):
    n = np.isnan(a)
    return np.array_equal(n, np.isnan(b)) and np.array_equal(a[~n].view(np.int64), b[~n].view(np.int64))


def test_seed(libs):
    d = torch.empty(1 << 23, dtype=torch.int32, device="cuda")
    assert libs[0].fm_seed_device(ctypes.c_void_p(d.data_ptr())) == 0
    assert int(d.abs().max()) <= 1


@pytest.mark.parametrize("name", list(CASES))
def test_functions(libs, name):
    fn, xs, _ = CASES[name]
    xs = np.concatenate([xs, SPECIAL])
    got, want = device(libs, fn, xs)[0], host(libs, fn, xs)
    if fn == 4:
        f = ~np.isnan(want)
        assert np.array_equal(np.isnan(got), ~f)
        assert (np.abs(got[f].view(np.int64) - want[f].view(np.int64)) <= 1).all()
    else:
        assert same(got, want)


@pytest.mark.parametrize("fn,single", [(9, 2), (10, 0)])
def test_pairs(libs, fn, single):
    xs = np.concatenate([SPECIAL] + [x for f, x, _ in CASES.values() if f == single])
    ys = np.random.default_rng(3).permutation(xs)
    q, q2 = device(libs, fn, xs, ys)
    assert same(q, host(libs, single, xs)) and same(q2, host(libs, single, ys))


@pytest.mark.parametrize("ea,eb", [(0, 0), (500, -500), (-1022, 0), (-1022, 1), (1023, -1), (0, 1023), (0, 1022),
                                   (0, -1022), (512, -511), (-511, 512)])
def test_quotients_and_roots(libs, ea, eb):
    """IEEE results, from numpy; the reciprocal square root from the host build."""
    rng = np.random.default_rng(abs(ea) * 7 + abs(eb))
    m = significands(rng, 2000)
    a = np.concatenate([np.ldexp(rng.permutation(m), ea), np.repeat(SPECIAL, SPECIAL.size)])
    b = np.concatenate([np.ldexp(m, eb), np.tile(SPECIAL, SPECIAL.size)])
    with np.errstate(all="ignore"):
        assert same(device(libs, 3, b)[0], 1.0 / b)
        assert same(device(libs, 6, a, b)[0], a / b)
        q, q2 = device(libs, 7, a, b)
        assert same(q, a / b) and same(q2, (2.5 * a) / b)
        assert same(device(libs, 8, a)[0], np.sqrt(a))
    assert same(device(libs, 5, a)[0], host(libs, 5, a))
