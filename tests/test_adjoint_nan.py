"""NaN states in the hand-written adjoint of ice_adjust (host build): what is
skipped where it is zero is not skipped where it is NaN."""
import numpy as np
import pytest

from ice3gb.constants import build_table
from test_adjoint_host import IN, OUT, _state, lib, vjp  # noqa: F401


@pytest.mark.parametrize("field", ["th", "exn", "rho_dry_ref", "rv"])
def test_nan_reaches_the_cloud_fraction_gradient(lib, field):  # noqa: F811
    """Without mass-flux clouds the gradient of cf_mf still carries the
    thresholds, NaN where the density or the temperature is."""
    table = build_table(table="phyex")
    x = {k: np.array(v, dtype=np.float64) for k, v in _state(16, 5).items() if k in IN}
    n = x["th"].size
    x = {k: np.resize(v.ravel(), n).copy() for k, v in x.items()}
    bad = np.arange(n) % 7 == 0
    x[field][bad] = np.nan
    rng = np.random.default_rng(1)
    gx = vjp(lib, table, x, {k: rng.normal(size=n) for k in OUT})
    assert np.isnan(gx["cf_mf"][bad]).all()
    assert np.isfinite(gx["cf_mf"][~bad]).all()
