"""A NaN pressure or potential temperature in the adjoint of the sedimentation:
at a level where cloud droplets fall (content or incoming flux above the
threshold) its gradient is NaN, whichever of the two flux bounds the forward
took; at a level without any it is 0."""
import numpy as np
import pytest

from ice3gb.constants import build_table
from test_adjoint_host import INPR, SRC, _sed_state, sed_vjp, sedlib  # noqa: F401

DT = 50.0


def _nan_state(field, nij=64, seed=7):
    x = {k: np.array(v, dtype=np.float64) for k, v in _sed_state(nij, seed).items()}
    bad = np.random.default_rng(seed).random(x["pabs"].shape) < 0.05
    x[field][bad] = np.nan
    rng = np.random.default_rng(seed + 1)
    g = {k: rng.standard_normal(bad.shape) for k in SRC}
    g.update({k: rng.standard_normal(bad.shape[1]) for k in INPR})
    return x, bad, g


def _check(table, x, bad, grad, inflow):
    """inflow: the cloud flux entering each level from above."""
    cloud = x["rcs"] * DT > table.values["C_RTMIN"]
    assert (bad & cloud).sum() > 50
    assert np.isnan(grad[bad & cloud]).all()
    assert (grad[~cloud & (inflow == 0.0)] == 0.0).all()


@pytest.mark.parametrize("field", ["pabs", "tht"])
@pytest.mark.parametrize("fortran", [True, False])
def test_host_sweep(sedlib, field, fortran):  # noqa: F811
    """The inflow is 0 for certain where no level above holds cloud."""
    table = build_table(table="phyex" if fortran else "jax")
    x, bad, g = _nan_state(field)
    above = np.cumsum((x["rcs"] > 0.0)[::-1], axis=0)[::-1] - (x["rcs"] > 0.0)
    _check(table, x, bad, sed_vjp(sedlib, table, x, g, fortran)[field], above)


@pytest.mark.gpu
@pytest.mark.parametrize("field", ["pabs", "tht"])
@pytest.mark.parametrize("semantics", ["phyex", "jax"])
def test_kernel(field, semantics):
    import torch

    from ice3gb import Sedimentation
    from ice3gb.autodiff import sedimentation
    sed = Sedimentation(table=semantics, semantics=semantics)
    x, bad, g = _nan_state(field)
    t = {k: torch.as_tensor(v).cuda().requires_grad_() for k, v in x.items()}
    out = sedimentation(sed, DT, **t)
    sum((out[k] * torch.as_tensor(g[k]).cuda()).sum() for k in SRC + INPR).backward()
    flux = out["fpr_c"].detach().cpu().numpy()
    _check(sed.table, x, bad, t[field].grad.cpu().numpy(), np.concatenate([flux[1:], np.zeros((1, flux.shape[1]))]))
