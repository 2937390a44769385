"""The MTHINC fluxes (solphi_mthinc1.f) on both sides of the steepness where their FP64 form
changes, and for profiles the wrong way round, against the oracle."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("bet", [-2.0, -0.5, 0.0, 3.99, 4.0, 4.01, 6.0])
def test_dropin_fluxes(orc, fmf_lib, bet):
    """Random normals of lengths across the band test's limit at every steepness, phi over
    (0, 1) with its ends; beta <= 0 has every cell in the band.  Up to 4.01 a flux differs
    by a few roundings of exp and cosh (1e-12 of the largest); at 6 overshooting cells
    multiply them, by 1e5 at most in 400 000 random cells: 1e-9."""
    ni, nj, nk = 32, 16, 16
    cfg = C.Config("steepness", ni, nj, nk, 2.0, 1.0, 1.0, dt=1e-3, steps=1)
    rng = np.random.default_rng(11)
    shape = cfg.shape
    long = 10.0 ** np.repeat(rng.uniform(-6, 1, shape[0] // 2), 2)[:, None, None]
    grads = [long * rng.normal(size=shape) / cfg.dx for _ in range(3)]
    phi = rng.uniform(0, 1, shape)
    ends = rng.uniform(size=shape) < 0.3
    phi[ends] = 10.0 ** rng.uniform(-8, -1, ends.sum())
    flip = rng.uniform(size=shape) < 0.5
    phi[flip] = 1.0 - phi[flip]
    vel = [0.2 * cfg.dx / cfg.dt * rng.uniform(-1, 1, shape) for _ in range(3)]
    res = []
    fmf_lib.fmf_set_mode(capi.FMF_COHERENT)
    try:
        for L, name in ((orc.lib(), "orc_solphi_mthinc1"), (fmf_lib, "solphi_mthinc1_")):
            out = [np.zeros(shape) for _ in range(3)]
            arrays = [np.ascontiguousarray(a) for a in [phi] + grads + vel] + out
            getattr(L, name)(*[capi.I(n) for n in (ni, nj, nk)], *[capi.D(1 / d) for d in (cfg.dx, cfg.dy, cfg.dz)],
                             capi.D(cfg.dt), capi.D(bet), *[ctypes.c_void_p(a.ctypes.data) for a in arrays])
            res.append(out)
        assert fmf_lib.fmf_last_error() == 0
    finally:
        fmf_lib.fmf_set_mode(capi.FMF_RESIDENT)
    for a, b in zip(*res):
        assert np.isfinite(a).all() and np.abs(a).max() > 0.05
        assert np.abs(a - b).max() <= (1e-9 if bet > 4.5 else 1e-12) * np.abs(a).max()


@pytest.mark.parametrize("bet", [4.0, 4.01, 6.0])
def test_step(orc, fmf_lib, bet):
    """One step of the fused solver with a randomly wrinkled interface; the bounds as above
    for the sum of six fluxes, with phi at most 1."""
    ni, nj, nk = 64, 16, 32
    cfg = C.get("couette128", ni=ni, nj=nj, nk=nk, bet_mthinc=bet, dt=1e-4)
    st = C.raw_state(cfg)
    rng = np.random.default_rng(5)
    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in cfg.shape], indexing="ij")
    for c in range(3):
        f = np.sin(2 * np.pi * (x / ni + 0.3 * c)) + np.cos(2 * np.pi * z / nk) * np.sin(np.pi * y / nj)
        st[c] = st[c + 3] = 0.1 * cfg.dx / cfg.dt * f
    d = np.abs(x - 0.5 * ni - 2) - ni / 4 + 2 * np.sin(2 * np.pi * z / nk) + 0.8 * rng.standard_normal(cfg.shape)
    st[9] = np.clip(0.5 * (1 + np.tanh(d / 1.2)), 1e-7, 1 - 1e-7)
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
    assert np.abs(a - b).max() <= (1e-9 if bet > 4.5 else 1e-13)


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_step_random(orc, fmf_lib, seed):
    """beta = 8, phi random from cell to cell with three tenths near 0 and two near 1, so that
    thousands of cells overshoot: the parity of 1e-10 with a factor of five for the cell
    that multiplies its roundings most."""
    ni, nj, nk = 128, 32, 64
    cfg = C.get("couette128", ni=ni, nj=nj, nk=nk, bet_mthinc=8.0, dt=1e-4)
    st = C.raw_state(cfg)
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in cfg.shape], indexing="ij")
    for c in range(3):
        f = np.sin(2 * np.pi * (x / ni + 0.3 * c)) + np.cos(2 * np.pi * z / nk) * np.sin(np.pi * y / nj)
        st[c] = st[c + 3] = 0.1 * cfg.dx / cfg.dt * f
    phi, kind = rng.uniform(0, 1, cfg.shape), rng.uniform(size=cfg.shape)
    phi = np.where(kind < 0.3, 10.0 ** rng.uniform(-8, -0.3, cfg.shape), phi)
    phi = np.where((kind > 0.3) & (kind < 0.5), 1 - 10.0 ** rng.uniform(-8, -0.3, cfg.shape), phi)
    st[9] = phi
    C.periodic(st[9], cfg)
    s = orc.Solver(cfg)
    orc.lib().orc_init_bc(s.ws, s._ptrs(st), *[orc.P(w) for w in s.walls])
    g = capi.Stepper(cfg)
    g.upload(st)
    g.step(1)
    got = g.get_state()
    g.close()
    s.step(st, 1)
    assert np.abs(C.interior(got[9]) - C.interior(st[9])).max() <= 5e-10


def test_reversed_profile_returns(fmf_lib):
    """beta = -8, where the truncation threshold is 1: a step ends (in a process of its own)
    and phi stays in [0, 1]."""
    code = """
import sys
sys.path.insert(0, {pkg!r})
from fmf import capi
from fmf import config as C
g = capi.Stepper(C.get("couette32", bet_mthinc=-8.0))
g.upload(g.initial_state())
g.step(2)
phi = C.interior(g.get_state()[9])
assert phi.min() >= 0.0 and phi.max() <= 1.0
""".format(pkg=os.path.join(ROOT, "fel-multi-phase-flow_gb300"))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
