"""Results do not depend on how a call is spread over the GPU: rain_ice on a
few columns (blocks of one to sixteen warps, a partial cluster of the ordering,
a partial warp of sedimentation columns) gives bit for bit the values that the
same columns get inside a larger call.  evap3d is left out: the last pass of
the whole call decides it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def big():
    from ice3gb import RainIce
    from ice3gb.state import make_state, rain_ice_state
    state = rain_ice_state(make_state(2400, 90, seed=5, precip=True, device="cuda"))
    ri = RainIce()
    return ri, state, ri(state, 50.0, with_fluxes=True)


@pytest.mark.parametrize("nij", [1, 2, 31, 33, 54, 55, 108, 433, 865, 1457])
def test_columns_of_a_larger_call(big, nij):
    ri, state, (new, diag) = big
    lo = 2400 - nij                                   # the last columns, an odd offset for odd nij
    part = {k: v[..., lo:].contiguous() for k, v in state.items()}
    n2, d2 = ri(part, 50.0, with_fluxes=True)
    for k in ("ci_t", "ths", "rvs", "rcs", "rrs", "ris", "rss", "rgs"):
        assert torch.equal(n2[k], new[k][..., lo:]), k
    for k in ("rainfr", "inprc", "inprr", "inpri", "inprs", "inprg", "fpr_c", "fpr_r", "fpr_i", "fpr_s", "fpr_g"):
        assert torch.equal(d2[k], diag[k][..., lo:]), k
