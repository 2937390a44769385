"""The viscous solve of a small grid in one launch (a thread-block cluster that applies
the stop rule itself) against the host-side rule over separate launches."""
import numpy as np
import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.FMF_FP64, capi.FMF_MIXED, capi.FMF_FP64E])
@pytest.mark.parametrize("shape", [(16, 8, 8), (32, 32, 16), (16, 64, 16), (64, 32, 16)])
def test_one_launch_solve_matches_host_rule(fmf_lib, monkeypatch, precision, shape):
    """From 1024 cells to the largest the cluster takes (2^14 in FP64, 2^15 in FP32; FP64 at
    2^15 runs the separate launches on both sides): the same state bit for bit and the same
    iteration counts over 10 steps in calls of one and of several, then at the iteration cap
    and back."""
    ni, nj, nk = shape
    cfg = C.get("couette256", ni=ni, nj=nj, nk=nk)
    g = capi.Stepper(cfg)
    st = g.initial_state()
    g.close()
    res = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("FMF_DEVICE_LOOP", mode)
        S = capi.Stepper(cfg, precision=precision)
        monkeypatch.delenv("FMF_DEVICE_LOOP")
        try:
            S.upload(st)
            its = []
            for n in (1, 7, 2):
                S.step(n)
                its += list(S.sor_iterations())
            S.set_sor(1e-300, 4)
            assert capi.lib().fmf_ctx_step(S.h, 2) == capi.FMF_ERR_ITER_CAP
            its += list(S.sor_iterations())
            S.set_sor(1e-3, 21)
            S.step(2)
            its += list(S.sor_iterations())
            res[mode] = (S.get_state(), its)
        finally:
            S.close()
    (a, ia), (b, ib) = res["0"], res["1"]
    assert ia == ib
    assert ia[10:12] == [4, 4]
    assert np.array_equal(a, b)


def test_one_launch_solve_reports_nonfinite(fmf_lib):
    """A velocity that is NaN ends the solve after its first iteration with the status the
    host-side rule gives."""
    cfg = C.get("couette32", ni=16, nj=8, nk=8)
    g = capi.Stepper(cfg)
    st = g.initial_state()
    st[0, 6, 6, 8] = np.nan
    g.upload(st)
    assert capi.lib().fmf_ctx_step(g.h, 2) == 3  # FMF_ERR_NONFINITE
    assert list(g.sor_iterations()) == [1, 1]
    g.close()
