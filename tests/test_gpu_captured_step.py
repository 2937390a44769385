"""The captured step (two branches beside the transport; small grids: the whole solve in one
launch) against the same kernels one by one on one stream (FMF_GRAPHS=0)."""
import numpy as np
import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu
PRECISIONS = [capi.FMF_FP64, capi.FMF_MIXED, capi.FMF_FP64E]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("shape", [(16, 8, 8), (16, 8, 4), (32, 8, 64), (64, 32, 32), (128, 64, 16)])
def test_captured_matches_eager(fmf_lib, monkeypatch, precision, shape):
    """Grids with and without the fused surface tension, the one-pass refresh and the
    one-launch solve; steps that continue the one before and steps on a new state."""
    ni, nj, nk = shape
    cfg = C.get("couette128", ni=ni, nj=nj, nk=nk)
    g = capi.Stepper(cfg)
    st = g.initial_state()
    g.close()
    rng = np.random.default_rng(1)
    res = {}
    other = st.copy()
    other[:6] += 1e-3 * rng.standard_normal(other[:6].shape)
    for mode in ("0", "1"):
        monkeypatch.setenv("FMF_GRAPHS", mode)
        S = capi.Stepper(cfg, precision=precision)
        monkeypatch.delenv("FMF_GRAPHS")
        out, its = [], []
        for state in (st, other, st):
            S.upload(state)
            for n in (1, 4):
                S.step(n)
                its += list(S.sor_iterations())
                out.append(S.get_state())
        S.close()
        res[mode] = (out, its)
    assert res["0"][1] == res["1"][1]
    for a, b in zip(res["0"][0], res["1"][0]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("shape", [(16, 8, 8), (32, 32, 16), (64, 32, 16)])
def test_small_solve_is_one_launch(fmf_lib, precision, shape):
    """Up to 2^14 cells (mixed: 2^15) a step launches the same number of kernels whether its
    solve takes 3 iterations or 9; beyond, more."""
    ni, nj, nk = shape
    S = capi.Stepper(C.get("couette256", ni=ni, nj=nj, nk=nk), precision=precision)
    S.upload(S.initial_state())
    S.step(2)
    L = capi.lib()
    launched = []
    for cap in (3, 9):
        S.set_sor(1e-300, cap)
        before = L.fmf_kernel_launches()
        assert L.fmf_ctx_step(S.h, 1) == capi.FMF_ERR_ITER_CAP
        launched.append(L.fmf_kernel_launches() - before)
        assert list(S.sor_iterations()) == [cap]
    S.close()
    small = ni * nj * nk <= (1 << 15 if precision == capi.FMF_MIXED else 1 << 14)
    assert (launched[0] == launched[1]) == small, launched
