"""The transposed viscous sweep where a point's adjoint and those of its periodic images
cancel exactly: the refresh gives the images the point's own value, so their adjoints add
up at the point, and a sum of 0 leaves nothing behind."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fel-multi-phase-flow_gb300", "csrc")
SHAPE = (16, 16, 16)


@pytest.fixture(scope="module")
def solve(fmf_lib, tmp_path_factory):
    from fmf import build
    so = str(tmp_path_factory.mktemp("sor_T") / "sor_T_check.so")
    subprocess.run([build.nvcc()] + build.ARCH +
                   ["-std=c++17", "-O2", "--extended-lambda", "-Xcompiler", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "sor_T_check.cu"), "-o", so, "-L", build.OUT, "-lfmf",
                    "-Xlinker", "-rpath=" + build.OUT], check=True)
    fn = ctypes.CDLL(so).sor_T_check
    fn.argtypes = [ctypes.c_int] * 3 + [ctypes.c_void_p] * 2
    return fn


@pytest.mark.parametrize("point", [(15, 7, 4), (5, 5, 2), (15, 9, 14), (16, 6, 3), (1, 6, 7), (13, 10, 1), (3, 8, 15),
                                   (2, 5, 5), (1, 6, 8)])
def test_cancelling_images(solve, point):
    """A point of w, the component the transposed cycle starts with, in each of the three
    colour pairs whose images the sweep gathers, next to an x face, a z face and both; every
    other adjoint is 0, and so is every gradient."""
    ni, nj, nk = SHAPE
    n = (ni + 6) * (nj + 6) * (nk + 6)
    rng = np.random.default_rng(3)
    fields = rng.uniform(0.5, 1.0, (55, nk + 6, nj + 6, ni + 6))
    fields[4:10] *= 1e-3  # A and B of the sweeps
    fields[10:13] = 0.0   # the adjoint of the solve's result
    i, j, k = point
    ix = i + ni if i <= 3 else (i - ni if i >= ni - 2 else None)
    kz = k + nk if k <= 3 else (k - nk if k >= nk - 2 else None)
    images = {(i, k): 1.75}
    if ix is not None and kz is not None:
        images.update({(ix, k): -1.0, (i, kz): -0.5, (ix, kz): -0.25})
    elif ix is not None:
        images[(ix, k)] = -1.75
    else:
        images[(i, kz)] = -1.75
    assert len(images) > 1
    for (a, c), v in images.items():
        fields[12, c + 2, j + 2, a + 2] = v
    wallc = rng.uniform(0.5, 1.0, 4 * (nk + 6) * (ni + 6))
    args = np.concatenate([fields.ravel(), wallc])
    out = np.full(10 * n, np.nan)
    assert solve(ni, nj, nk, args.ctypes.data, out.ctypes.data) == 0
    assert np.count_nonzero(out) == 0
