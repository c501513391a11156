"""A zero density without mass-flux clouds (host build of ia_point_vjp): the
autoconversion threshold of the mass-flux cloud is infinite and its gradients
are NaN, as with the mass-flux update of other points; finite at the points with
an ordinary density."""
import numpy as np

from ice3gb.constants import build_table
from test_adjoint_host import IN, OUT, _state, lib, vjp  # noqa: F401


def test_threshold_gradients_are_nan(lib):  # noqa: F811
    table = build_table(table="phyex")
    x = {k: np.array(v, dtype=np.float64) for k, v in _state(16, 5).items() if k in IN}
    n = x["th"].size
    x = {k: np.ascontiguousarray(np.broadcast_to(v, x["th"].shape)).ravel().copy() for k, v in x.items()}
    bad = np.arange(n) % 7 == 0
    x["rho_dry_ref"][bad] = 0.0
    rng = np.random.default_rng(1)
    g = vjp(lib, table, x, {k: rng.normal(size=n) for k in OUT})
    for k in ("cf_mf", "rc_mf", "rho_dry_ref"):
        assert np.isnan(g[k][bad]).all() and np.isfinite(g[k][~bad]).all(), k
