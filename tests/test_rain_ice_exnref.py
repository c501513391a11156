"""A zero reference Exner function in rain_ice (host build of the point code):
the latent heat factors are infinite, and the nucleation that does not happen
adds 0 times infinity to the source of theta, NaN where the oracle has it.
(Where it happens the source is infinite, as the correction of negative sources
is skipped where it moves nothing.)"""
import ctypes

import numpy as np

from ice3gb.constants import build_table
from test_rain_ice_host import DT, host_lib  # noqa: F401


def test_theta_source_is_nan_where_the_oracles_is(host_lib):  # noqa: F811
    import oracle
    from ice3gb import _abi
    from ice3gb.state import make_state
    from test_gpu_rain_ice import _abi_rain_ice_state
    nij, nk = 64, 90
    t = build_table(table="phyex")
    x = _abi_rain_ice_state({k: v.numpy() for k, v in make_state(nij, nk, seed=0, precip=True).items()})
    x = {k: np.array(v, dtype=np.float64) for k, v in x.items()}
    x["exnref"].ravel()[::11] = 0.0
    sed = oracle.sedimentation(t, x, DT, True)
    keep = {k: np.array(x[k]) for k in ("exn", "dzz", "rhodref", "exnref", "pabs", "cldfr", "sigs", "tht", "rvt", "rct",
                                        "rrt", "rit", "rst", "rgt", "sea", "town", "cit", "hlc_hrc", "hlc_hcf",
                                        "hli_hri", "hli_hcf", "ths", "rvs")}
    keep.update({k: np.array(sed[k]) for k in ("rcs", "rrs", "ris", "rss", "rgs")})
    keep.update({k: np.zeros((nk, nij)) for k in ("evap3d", "rainfr")})
    f = _abi.RainIceFields()
    for k, v in keep.items():
        setattr(f, k, v.ctypes.data)
    keys = np.zeros(nij * nk, dtype=np.uint32)
    assert host_lib.rain_ice_points_host(ctypes.byref(t.consts), ctypes.byref(t.luts), nij, nk, ctypes.c_double(DT), 256,
                                         ctypes.byref(f), keys.ctypes.data_as(ctypes.c_void_p)) == 0
    ref = oracle.rain_ice(t, x, DT)[0]
    still = ref["cit"] == x["cit"]                     # no nucleation
    want = np.isnan(ref["ths"]) & still
    assert want.sum() > 100
    assert np.array_equal(np.isnan(keep["ths"]) & still, want)
