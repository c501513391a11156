"""An infinite temperature without mass-flux clouds (host build of ia_point): the
mass-flux update adds 0 times the infinite latent heat to theta's source, which
is NaN, as the oracle has it."""
import numpy as np
import pytest

from ice3gb.constants import build_table
from test_adjoint_host import DT, IN, _state, forward, lib  # noqa: F401


@pytest.mark.parametrize("field", ["th", "exn"])
@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("mode", [0.0, 1.0, 3.0])
def test_theta_source_is_nan(lib, field, value, mode):  # noqa: F811
    import oracle
    table = build_table(table="phyex", overrides={"FRAC_ICE_ADJUST": mode})
    x = {k: np.array(v, dtype=np.float64) for k, v in _state(16, 5).items() if k in IN}
    x["sigqsat"] = np.ascontiguousarray(np.broadcast_to(x["sigqsat"], x["th"].shape))
    x[field].ravel()[::7] = value
    got, ref = forward(lib, table, x)["ths"], oracle.ice_adjust(table, x, DT)["ths"].ravel()
    assert np.isnan(ref[::7]).all()
    assert np.array_equal(np.isnan(got), np.isnan(ref))
