"""NaN states in the rain_ice point code (host build): the decisions taken in
FP32 or on bit patterns have to come out as the FP64 comparisons they stand
for, which a NaN makes false."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from ice3gb.constants import build_table

HERE = os.path.dirname(os.path.abspath(__file__))


def _build(tmp_path_factory, name):
    out = tmp_path_factory.mktemp(name) / f"lib{name}.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(HERE, "..", "include"), os.path.join(HERE, f"{name}.cpp"), "-o", str(out)], check=True)
    return ctypes.CDLL(str(out))


@pytest.fixture(scope="module")
def pdf(tmp_path_factory):
    return _build(tmp_path_factory, "rain_ice_nan_host")


@pytest.mark.parametrize("t", [np.nan, np.inf, 200.0, 233.15, 253.15, 273.15])
def test_soft_ice_threshold_is_the_full_one(pdf, t):
    """Equality: the indicator is 0 or 1 in both forms."""
    table = build_table(table="phyex")
    rit = np.concatenate([10.0 ** np.linspace(-12, -2, 400), [float(table.consts.CRIAUTI)]])
    tt, soft, full = np.full(rit.size, t), np.empty(rit.size), np.empty(rit.size)
    pdf.ice_high_host(ctypes.byref(table.consts), ctypes.c_long(rit.size),
                      *[a.ctypes.data_as(ctypes.c_void_p) for a in (tt, rit, soft, full)])
    assert (soft == full).all()


@pytest.mark.parametrize("nan", [np.nan, -np.nan])
def test_crossing_is_the_product_test(pdf, nan):
    """Equality, over all triples of values around a potential temperature,
    infinities and NaN."""
    v = np.array([250.0, 273.16, np.nextafter(273.16, 0), np.nextafter(273.16, 300), 290.0, 0.0, -1.0, np.inf, -np.inf, nan])
    a, b, z = (np.ascontiguousarray(g.ravel()) for g in np.meshgrid(v, v, v))
    out = np.empty(a.size, dtype=np.int32)
    pdf.crosses_host(ctypes.c_long(a.size), *[g.ctypes.data_as(ctypes.c_void_p) for g in (a, b, z, out)])
    with np.errstate(invalid="ignore"):
        assert (out.astype(bool) == ((a - z) * (b - z) < 0)).all()
