"""The recorded forward step's viscous solve on a small grid at an iteration cap beyond the
100 000 that one launch runs at most: fmf_adj_set_solver takes it, and the solve reaches it."""
import pytest

from fmf import config as C

pytestmark = pytest.mark.gpu


def test_cap_beyond_one_launch(fmf_lib, monkeypatch):
    """A tolerance no residual meets, so that the count is the cap (a solve that ends there
    counts one more)."""
    from fmf.adjoint import Adjoint

    cfg = C.get("couette128", ni=16, nj=8, nk=8)
    monkeypatch.setenv("FMF_ADJ_RECORD_ALL", "1")
    adj = Adjoint(cfg, sor_tol=1e-300, sor_max=100003, adj_tol=1e-10, adj_max=10)
    monkeypatch.delenv("FMF_ADJ_RECORD_ALL")
    adj.forward(1, C.raw_state(cfg), [w.copy() for w in C.wall_arrays(cfg)])
    assert adj.iterations()[0] == 100004
    adj.close()
