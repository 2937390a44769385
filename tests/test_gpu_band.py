"""The FP64 interface band (Newton offset and swept-volume fluxes of solphi_mthinc1.f)
through one step of the fused solver, against the oracle."""
import numpy as np
import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bet", [0.5, 2.0, 3.5])
@pytest.mark.parametrize("cfl", [1e-3, 0.2])
def test_band_fluxes(orc, fmf_lib, bet, cfl):
    """Interface steepness from one whose sigmoids are nearly flat to one whose Newton steps
    leave the range of the tabulated exponential, swept volumes from thin to a fifth of a
    cell, a randomly wrinkled interface with phi from 1e-7 to 1 - 1e-7 in
    the band (cells whose ten Newton steps converge and cells whose do not).  A flux is a
    mean of eight sigmoids, each a few roundings off on either side, times a Courant
    number below one; phi is at most 1, so 1e-13 covers the differences of six of them."""
    ni, nj, nk = 64, 16, 32
    cfg = C.get("couette128", ni=ni, nj=nj, nk=nk, bet_mthinc=bet, dt=1e-4)
    st = C.raw_state(cfg)
    rng = np.random.default_rng(int(10 * bet))
    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in cfg.shape], indexing="ij")
    speed = cfl * cfg.dx / cfg.dt
    for c in range(3):
        f = np.sin(2 * np.pi * (x / ni + 0.3 * c)) + np.cos(2 * np.pi * z / nk) * np.sin(np.pi * y / nj)
        st[c] = st[c + 3] = 0.5 * speed * f
    d = np.abs(x - 0.5 * ni - 2) - ni / 4 + 2 * np.sin(2 * np.pi * z / nk) + 0.8 * rng.standard_normal(cfg.shape)
    phi = 0.5 * (1 + np.tanh(d / 1.2))
    st[9] = np.clip(phi, 1e-7, 1 - 1e-7)
    C.periodic(st[9], cfg)
    s = orc.Solver(cfg)
    orc.lib().orc_init_bc(s.ws, s._ptrs(st), *[orc.P(w) for w in s.walls])
    g = capi.Stepper(cfg)
    g.upload(st)
    g.step(1)
    got = g.get_state()
    g.close()
    s.step(st, 1)
    a, b = C.interior(got[9]), C.interior(st[9])
    assert ((b > 0) & (b < 1)).sum() > 1000
    assert np.abs(a - b).max() <= 1e-13
