"""The transposed viscous solve with the swept component's images gathered by the sweep,
against the transposed refresh before every sweep (FMF_REFRESH_ORDERED): the same J and,
up to the order of the additions, the same gradients."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import sys
sys.path.insert(0, {pkg!r})
import numpy as np
from fmf import config as C
from fmf.adjoint import Adjoint
cfg = C.get("couette128", ni={ni}, nj={nj}, nk={nk})
adj = Adjoint(cfg, sor_tol=1e-13, sor_max=300, adj_tol=1e-13, adj_max=400)
J, g = adj.rollout(3, C.raw_state(cfg), [w.copy() for w in C.wall_arrays(cfg)])
np.savez({path!r}, J=J, **{{"g%d" % i: a for i, a in enumerate(g)}})
"""


def _run(tmp_path, ordered, ni, nj, nk):
    path = str(tmp_path / f"{int(ordered)}.npz")
    env = dict(os.environ)
    env.pop("FMF_REFRESH_ORDERED", None)
    if ordered:
        env["FMF_REFRESH_ORDERED"] = "1"
    code = SCRIPT.format(pkg=os.path.join(ROOT, "fel-multi-phase-flow_gb300"), ni=ni, nj=nj, nk=nk, path=path)
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(path)


@pytest.mark.parametrize("shape", [(16, 8, 8), (32, 8, 64), (128, 16, 8)])
def test_images_gathered_by_the_sweep(fmf_lib, tmp_path, shape):
    """The smallest one-pass grid, one thread row in x (16) and two (128)."""
    a = _run(tmp_path, False, *shape)
    b = _run(tmp_path, True, *shape)
    assert a["J"] == b["J"]
    for i in range(5):
        x, y = a[f"g{i}"], b[f"g{i}"]
        assert np.isfinite(x).all()
        assert np.abs(x - y).max() <= 1e-10 * max(np.abs(y).max(), 1e-300), i
