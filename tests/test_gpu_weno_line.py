"""The FP64 step's WENO5 (fmf_dev_weno5_fused, FMF_FP64), which walks lines of one to
32 points per thread, against the oracle's cal_advu_weno5.f:38-255."""
import numpy as np
import pytest

from fmf import capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,nk", [(4, 4, 4), (16, 8, 8), (32, 16, 16), (8, 256, 8), (64, 32, 32), (16, 16, 256),
                                      (128, 64, 64)])
@pytest.mark.parametrize("scale", [1.0, 1e-10])
def test_weno_line_against_oracle(orc, fmf_lib, ni, nj, nk, scale):
    """Grids from the smallest to one walked 32 points at a time, lines shorter than a
    warp and than a walk, on data with jumps, an exactly linear part, zeros (velocity
    sums that are 0) and noise, both signs of the velocity everywhere; at 1e-10 the
    reference's additive 1e-80 is as large as the weights.  Both sides take the same
    rounded differences D of the velocities; a term is at most |vel| dxi max|D| and the
    rearranged weights move it by some tens of roundings of D (1.1e-16 each), so each
    component agrees within 1e-13 of its largest value."""
    import torch

    shape = (nk + 6, nj + 6, ni + 6)
    rng = np.random.default_rng(ni + 7 * nj + 31 * nk)
    z, y, x = np.meshgrid(*[np.arange(n, dtype=float) for n in shape], indexing="ij")
    fields = []
    for c in range(3):
        f = np.sin(0.5 * x + c) * np.cos(0.4 * y) + 0.5 * np.sin(0.3 * z + 2 * c) + np.where(x > shape[2] / 2, 0.7, 0)
        f = np.where(y < 6, 0.05 * z - 0.1 * c, f)
        f = np.where((z > 3) & (z < 7) & (x < 12), 0.0, f)
        f = np.where(y > nj, rng.standard_normal(shape), f)
        fields.append(np.ascontiguousarray(f * scale))
    dxi, dyi, dzi = ni / 2.0, float(nj), nk * 1.5
    ref = [np.zeros(shape) for _ in range(3)]
    I, D, P = orc.I, orc.D, orc.P
    orc.lib().orc_cal_advu_weno5(I(ni), I(nj), I(nk), D(dxi), D(dyi), D(dzi), *[P(f) for f in fields],
                                 *[P(a) for a in ref])
    dev = [torch.from_numpy(f).cuda() for f in fields]
    got = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()  # the library runs on its own stream
    capi.check(fmf_lib.fmf_dev_weno5_fused(capi.FMF_FP64, ni, nj, nk, dxi, dyi, dzi, *[d.data_ptr() for d in dev],
                                           *[t.data_ptr() for t in got]), "weno5")
    assert fmf_lib.fmf_device_synchronize() == 0
    for a, b in zip(got, ref):
        m = np.abs(b).max()
        assert m > 0
        assert np.abs(a.cpu().numpy() - b).max() <= 1e-13 * m
