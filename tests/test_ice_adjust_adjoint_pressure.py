"""The pressure gradient of ice_adjust (host build of ia_point_vjp) is NaN where
the saturation's cotangent is: at an infinite temperature, whose
saturation pressure is 0, and at zero pressure, where the mixing ratio is 0 / 0;
finite at the other points."""
import numpy as np
import pytest

from ice3gb.constants import build_table
from test_adjoint_host import IN, OUT, _state, lib, vjp  # noqa: F401


@pytest.mark.parametrize("field,value", [("th", np.inf), ("exn", np.inf), ("th", -np.inf), ("pabs", 0.0)])
@pytest.mark.parametrize("mode", [0.0, 1.0, 3.0])
def test_pressure_gradient_is_nan(lib, field, value, mode):  # noqa: F811
    table = build_table(table="phyex", overrides={"FRAC_ICE_ADJUST": mode})
    x = {k: np.array(v, dtype=np.float64) for k, v in _state(16, 5, mf=True).items() if k in IN}
    n = x["th"].size
    x = {k: np.ascontiguousarray(np.broadcast_to(v, x["th"].shape)).ravel().copy() for k, v in x.items()}
    bad = np.arange(n) % 7 == 0
    x[field][bad] = value
    rng = np.random.default_rng(1)
    g = vjp(lib, table, x, {k: rng.normal(size=n) for k in OUT})["pabs"]
    assert np.isnan(g[bad]).all() and np.isfinite(g[~bad]).all()
