"""The colour-pair sweeps and momentum factors of warps in one fluid (2^21 cells and more,
nine tenths of them away from the interface) against the oracle: a drop in a box of
256x128x64."""
import numpy as np
import pytest

from fmf import capi
from fmf import config as C
from test_gpu_step_shapes import _start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.FMF_FP64, capi.FMF_FP64E])
def test_flat_sweeps(orc, fmf_lib, precision):
    """Two steps (the second's densities are the first's phi, exactly 0 or 1 away from the
    interface), every field with its halos within the step's 1e-10 of the oracle."""
    cfg = C.get("droplet256", ni=256, nj=128, nk=64)
    s, st = _start(orc, cfg, 5)
    g = capi.Stepper(cfg, precision)
    g.upload(st)
    g.step(2)
    got = g.get_state()
    iters = g.sor_iterations()
    g.close()
    s.step(st, 2)
    phi = got[C.STATE_FIELDS.index("phin0")]
    assert ((phi == 0) | (phi == 1)).mean() > 0.93  # the share that switches the path on is 0.9
    assert iters == s.sor_iters
    for f, name in enumerate(C.STATE_FIELDS):
        err = np.abs(got[f] - st[f]).max() / max(np.abs(st[f]).max(), 1e-30)
        assert err <= 1e-10, (name, err)


def test_flat_sweeps_mixed(orc, fmf_lib):
    """The mixed-precision step on the same box: within its 1e-5 of the oracle."""
    cfg = C.get("droplet256", ni=256, nj=128, nk=64)
    s, st = _start(orc, cfg, 5)
    g = capi.Stepper(cfg, capi.FMF_MIXED)
    g.upload(st)
    g.step(2)
    got = g.get_state()
    g.close()
    s.step(st, 2)
    for f, name in enumerate(C.STATE_FIELDS):
        err = np.abs(got[f] - st[f]).max() / max(np.abs(st[f]).max(), 1e-30)
        assert err <= 1e-5, (name, err)
