"""A velocity that is not finite, far from the interface, where the transport's kernels skip
their arithmetic: phi of the two cells it is a face of, as the oracle's clip leaves it."""
import numpy as np
import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("i", [6, 32], ids=["phi0", "phi1"])
@pytest.mark.parametrize("comp", [0, 1, 2])
def test_phi_beside_it(orc, fmf_lib, comp, i, value):
    """phi is exactly 0 or 1 there after a first step; the solve reports the velocity."""
    cfg = C.get("couette32", ni=64, nj=32, nk=16)
    g = capi.Stepper(cfg)
    g.upload(g.initial_state())
    g.step(1)
    st = g.get_state()
    at = (8 + 2, 16 + 2, i + 2)
    assert st[9][at] == (0.0 if i == 6 else 1.0)
    st[comp][at] = value
    g.upload(st)
    assert capi.lib().fmf_ctx_step(g.h, 1) == 3  # FMF_ERR_NONFINITE
    got = g.get_state()[9]
    g.close()
    s = orc.Solver(cfg)
    s.step(st, 1)
    a, b = C.interior(got), C.interior(st[9])
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.nanmax(np.abs(a - b)) <= 1e-13
