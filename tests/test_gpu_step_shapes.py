"""The fused step against the oracle on grids of the shapes its kernels split
differently: lines shorter than a warp, one to many walks or planes per thread, thin in
every direction, with velocities of both signs and whole warps in flat regions."""
import numpy as np
import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu


def _start(orc, cfg, seed):
    st = C.raw_state(cfg)
    rng = np.random.default_rng(seed)
    z, y, x = np.meshgrid(*[np.arange(n) / n for n in cfg.shape], indexing="ij")
    for c in range(3):
        a, p = rng.uniform(0.05, 0.2, 3), rng.uniform(0, 6, 3)
        f = a[0] * np.sin(2 * np.pi * x + p[0]) + a[1] * np.cos(2 * np.pi * z + p[1]) * np.sin(np.pi * y)
        st[c] = st[c + 3] = f + a[2] * np.sin(2 * np.pi * (x + z) + p[2])
    s = orc.Solver(cfg)
    th, ze, l1, l2 = s.walls
    orc.lib().orc_init_bc(s.ws, s._ptrs(st), *[orc.P(w) for w in (th, ze, l1, l2)])
    return s, st


@pytest.mark.parametrize("ni,nj,nk", [(16, 4, 4), (16, 8, 64), (64, 8, 16), (32, 64, 8), (128, 16, 16), (64, 32, 64)])
@pytest.mark.parametrize("flow", ["couette128", "droplet256"])
@pytest.mark.parametrize("precision", [capi.FMF_FP64, capi.FMF_FP64E])
def test_step_shapes(orc, fmf_lib, ni, nj, nk, flow, precision):
    """Four steps (the first computes both velocity levels, the others carry one over),
    every field with its halos within the step's 1e-10 of the oracle, and the viscous
    iteration counts equal."""
    cfg = C.get(flow, ni=ni, nj=nj, nk=nk)
    if cfg.checker_cells:
        cfg.checker_cells = max(1, ni // 16)
    s, st = _start(orc, cfg, ni + nj + nk)
    g = capi.Stepper(cfg, precision)
    g.upload(st)
    g.step(4)
    got = g.get_state()
    iters = g.sor_iterations()
    g.close()
    s.step(st, 4)
    assert iters == s.sor_iters
    for f, name in enumerate(C.STATE_FIELDS):
        err = np.abs(got[f] - st[f]).max() / max(np.abs(st[f]).max(), 1e-30)
        assert err <= 1e-10, (name, err)
