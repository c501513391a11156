"""What the species' cotangents do to each other in the adjoint of the
sedimentation.  The cloud levels of a column whose rain cotangent is NaN at the
surface have a NaN pressure and theta gradient (the sum over the species that
they are formed from), the other columns none.  The layers are 2 km thick and
the scheme's rain speed at these contents is above 80 m/s, twice a layer per
step: the flux leaving a level is bounded by its content, and the NaN takes the
way through the speed of the flux that falls in, which the top level has not."""
import numpy as np
import pytest

from ice3gb.constants import build_table
from test_adjoint_host import INPR, SRC, _sed_state, sed_vjp, sedlib  # noqa: F401

DT = 50.0


def _case(nij=40, seed=3):
    x = {k: np.array(v, dtype=np.float64) for k, v in _sed_state(nij, seed).items()}
    x["dzz"][:] = 2000.0
    for k in ("rcs", "rrs"):
        x[k] = np.maximum(x[k], 1e-5 / DT)
    rng = np.random.default_rng(seed)
    g = {k: rng.standard_normal(x["dzz"].shape) for k in SRC}
    g.update({k: rng.standard_normal(nij) for k in INPR})
    bad = np.arange(nij) % 7 == 2
    g["inprr"][bad] = np.nan
    return x, g, bad


def _check(grad, bad):
    assert np.isnan(grad[:-1, bad]).all()
    assert np.isfinite(grad[-1]).all() and np.isfinite(grad[:, ~bad]).all()


@pytest.mark.parametrize("fortran", [True, False])
def test_host_sweep(sedlib, fortran):  # noqa: F811
    x, g, bad = _case()
    gx = sed_vjp(sedlib, build_table(table="phyex" if fortran else "jax"), x, g, fortran)
    _check(gx["pabs"], bad)
    _check(gx["tht"], bad)


@pytest.mark.gpu
@pytest.mark.parametrize("semantics", ["phyex", "jax"])
def test_kernel(semantics):
    import torch

    from ice3gb import Sedimentation
    from ice3gb.autodiff import sedimentation
    x, g, bad = _case()
    t = {k: torch.as_tensor(v).cuda().requires_grad_() for k, v in x.items()}
    out = sedimentation(Sedimentation(table=semantics, semantics=semantics), DT, **t)
    gx = torch.autograd.grad([out[k] for k in SRC + INPR], [t["pabs"], t["tht"]],
                             [torch.as_tensor(g[k]).cuda() for k in SRC + INPR])
    for v in gx:
        _check(v.cpu().numpy(), bad)
