"""The ice fraction of ice_adjust where it is decided on the high words of the
temperature (ia_point in ice_adjust_point.cuh, host build): at TMINMIX and
TMAXMIX, their neighbouring doubles and neighbouring high words, for mixed
ranges that are regular, reversed, empty and partly negative, against the
oracle; and NaN temperatures.  The outputs are NaN exactly where the oracle's
are (t = TMINMIX = TMAXMIX is 0/0; a fraction from the condensate keeps the
water finite at a NaN temperature).

Bound: the saturation pressure carries the error of an exponent of about 60
(a few 1e-14 relative), the sums a few ulp of the total water, so 1e-12 of the
total water leaves a factor of about 30."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from ice3gb.constants import build_table
from test_adjoint_host import DT, IN, _state, forward

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("ia") / "libia_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(HERE, "..", "include"), os.path.join(HERE, "ice_adjust_point_host.cpp"), "-o",
                    str(out)], check=True)
    return ctypes.CDLL(str(out))


def _at(temps, seed=5):
    """A state with the given temperatures (exn = 1) in its first points."""
    x = {k: np.array(v, dtype=np.float64) for k, v in _state(16, seed).items() if k in IN}
    shape = x["th"].shape
    x = {k: np.ascontiguousarray(np.broadcast_to(v, shape)).copy() for k, v in x.items()}
    n = len(temps)
    x["exn"].ravel()[:n] = 1.0
    x["th"].ravel()[:n] = temps
    return x, n


def _compare(got, ref, x, n, names):
    water = (x["rv"] + x["rc"] + x["ri"]).ravel()[:n]
    for k in names:
        g, r = got[k][:n], ref[k].ravel()[:n]
        assert (np.isnan(g) == np.isnan(r)).all(), k
        f = ~np.isnan(r)
        assert (np.abs(g[f] - r[f]) <= 1e-12 * water[f]).all(), k


@pytest.mark.parametrize("limits", [(253.16, 273.16), (200.0, 300.0), (300.0, 200.0), (250.0, 250.0), (-10.0, 273.16)])
@pytest.mark.parametrize("mode", [0.0, 1.0, 3.0])
def test_limits_match_oracle(lib, limits, mode):
    import oracle
    table = build_table(table="phyex", overrides={"TMINMIX": limits[0], "TMAXMIX": limits[1], "FRAC_ICE_ADJUST": mode})
    temps = []
    for t in [abs(v) if v > 0 else 240.0 for v in limits]:
        word = np.float64(t).view(np.int64)
        temps += list(np.array([word + d for d in (-2**33, -2**32, -2, -1, 0, 1, 2, 2**32, 2**33)]).view(np.float64))
    x, n = _at(temps)
    got, ref = forward(lib, table, x), oracle.ice_adjust(table, x, DT)
    _compare(got, ref, x, n, ("rv_out", "rc_out", "ri_out"))


@pytest.mark.parametrize("mode", [0.0, 1.0, 3.0])
@pytest.mark.parametrize("nan", [np.nan, -np.nan])
def test_nan_matches_oracle(lib, mode, nan):
    import oracle
    table = build_table(table="phyex", overrides={"FRAC_ICE_ADJUST": mode})
    x, n = _at([nan] * 8)
    _compare(forward(lib, table, x), oracle.ice_adjust(table, x, DT), x, n, ("t", "rv_out", "rc_out", "ri_out"))
