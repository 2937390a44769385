"""fmf_ctx_check_sor and stage 1 of fmf_ctx_time_stage on grids whose viscous solve is one
launch: they run that launch."""
import ctypes

import pytest

from fmf import capi
from fmf import config as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [capi.FMF_FP64, capi.FMF_MIXED, capi.FMF_FP64E])
def test_support_entries_take_the_step_s_solve(fmf_lib, precision):
    """The measured solve has the iterations of the next step and ends under its tolerance;
    twenty timed iterations are launches of one kernel each; neither changes what follows."""
    L = fmf_lib
    cfg = C.get("couette32")
    S, plain = capi.Stepper(cfg, precision=precision), capi.Stepper(cfg, precision=precision)
    st = S.initial_state()
    for g in (S, plain):
        g.upload(st)
        g.step(3)
    out = (ctypes.c_double * 5)()
    assert L.fmf_ctx_check_sor(S.h, out) == 0
    ms = ctypes.c_float()
    before = L.fmf_kernel_launches()
    assert L.fmf_ctx_time_stage(S.h, 1, 20, ctypes.byref(ms)) == 0
    assert 0 < ms.value < 5
    assert L.fmf_kernel_launches() - before <= 21 + 8
    for g in (S, plain):
        g.step(2)
    its = list(S.sor_iterations())
    assert its == list(plain.sor_iterations())
    assert out[0] == its[0] and 0 < out[1] <= 1e-3
    assert (S.get_state() == plain.get_state()).all()
    S.set_sor(1e-300, 9)  # at the cap
    assert L.fmf_ctx_check_sor(S.h, out) == 0 and out[0] == 9
    S.close()
    plain.close()
