"""The colour-pair sweeps at the grid sizes where their split changes, with the ghosts
written by the sweep, against the ordered plane kernels (FMF_REFRESH_ORDERED): the same
bits in FP64 and mixed precision."""
import numpy as np
import pytest

from test_gpu_refresh import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 8, 8), (16, 64, 16), (64, 64, 64), (128, 64, 128), (128, 128, 128)])
def test_sweep_ghosts_match_ordered_kernels(fmf_lib, tmp_path, shape):
    """2^10 to 2^21 cells: the colours split over blocks (FP64 below 2^18, FP32
    throughout), together (2^18), the ghosts refreshed apart in FP32 (2^20), four planes
    per thread (2^21)."""
    a = _run(tmp_path, "sweep", False, "droplet256", *shape, 3)
    b = _run(tmp_path, "ordered", True, "droplet256", *shape, 3)
    for key in ("fp64", "mixed"):
        assert np.isfinite(a[key]).all()
        assert np.array_equal(a[key], b[key]), (key, np.abs(a[key] - b[key]).max())
