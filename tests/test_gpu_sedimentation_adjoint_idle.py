"""Columns without any content next to one with an infinite density: the
adjoint's recomputed fluxes are NaN there (infinity times the zero content), as
in a warp that has something to move, and reach the gradients of rho and dz at
the level and the one below."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("semantics", ["phyex", "jax"])
@pytest.mark.parametrize("nij,col", [(64, 5), (33, 32)])
def test_infinite_density_without_content(semantics, nij, col):
    from ice3gb import Sedimentation
    from ice3gb.autodiff import sedimentation
    from test_adjoint_host import INPR, SRC, _sed_state
    x = {k: np.array(v[:12], dtype=np.float64)[:, :nij].copy() for k, v in _sed_state(64, 3).items()}
    for k in SRC:
        x[k][:] = 0.0
    x["rhodref"][6, col] = np.inf
    t = {k: torch.as_tensor(v).cuda().requires_grad_() for k, v in x.items()}
    out = sedimentation(Sedimentation(table=semantics, semantics=semantics), 50.0, **t)
    g = torch.autograd.grad(sum(out[k].sum() for k in SRC + INPR), [t["rhodref"], t["dzz"]])
    want = np.zeros((12, nij), dtype=bool)
    want[5:7, col] = True
    for v in g:
        assert np.array_equal(np.isnan(v.cpu().numpy()), want)
