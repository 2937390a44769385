"""The FP64 CSF force (fmf_dev_csf_fused, FMF_FP64) against the oracle's chain of
reference subroutines (main.f90:548-567)."""
import numpy as np
import pytest

from fmf import capi

pytestmark = pytest.mark.gpu


def _gpu(lib, ni, nj, nk, d, rho, sigma, phi):
    import torch

    t = torch.from_numpy(phi).cuda()
    f = [torch.zeros(phi.shape, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()  # the library runs on its own stream
    capi.check(lib.fmf_dev_csf_fused(capi.FMF_FP64, ni, nj, nk, *d, *rho, sigma, t.data_ptr(),
                                     *[q.data_ptr() for q in f]), "csf")
    assert lib.fmf_device_synchronize() == 0
    return [q.cpu().numpy() for q in f]


def _phi(ni, nj, nk, snap):
    z, y, x = np.meshgrid(*[np.arange(n + 6) - 2.5 for n in (nk, nj, ni)], indexing="ij")
    s = np.abs(x - 0.5 * ni) + 0.2 * y - 0.3 * z - 0.15 * ni
    phi = 0.5 * (1 + np.tanh(s / 1.5))
    if snap:  # exactly 0 and 1 outside the interface band
        phi = np.where(phi < 4.5e-5, 0.0, np.where(phi > 1 - 4.5e-5, 1.0, phi))
    return np.ascontiguousarray(phi)


@pytest.mark.parametrize("ni,nj,nk", [(32, 8, 4), (32, 16, 16), (64, 8, 64), (32, 32, 128), (128, 64, 64)])
@pytest.mark.parametrize("snap", [True, False])
def test_csf_fp64_against_oracle(orc, fmf_lib, ni, nj, nk, snap):
    """From the smallest grid to columns walked eight planes at a time, with whole warps
    in flat regions (snap) and with tails down to the last bit of 1.  phi is held to
    2^-53, so a gradient g carries 2^-53 dxi, its normal 2^-53 dxi / g and the force
    C kappa (phi(i+1) - phi(i)) dxi, C = 2 sigma/(rho_l + rho_g), about 2^-53 C dxi^2;
    with some hundred roundings on either side, 3e-14 C dxi^2."""
    dx, dy, dz = 2.0 / ni, 1.0 / nj, 1.25 / nk
    rhol, rhog, sigma = 10.0, 1.0, 0.7
    phi = _phi(ni, nj, nk, snap)
    sh = phi.shape
    I, D, P = orc.I, orc.D, orc.P
    N, inv = (I(ni), I(nj), I(nk)), (D(1 / dx), D(1 / dy), D(1 / dz))
    dya = np.full(nj + 6, 1 / dy)
    O = orc.lib()
    g = [np.zeros(sh) for _ in range(3)]
    O.orc_cal_grad_p2a(I(0), I(nj), *N, D(1 / dx), P(dya), D(1 / dz), P(phi), *[P(a) for a in g])
    rn = [np.zeros((3,) + sh) for _ in range(4)]
    for q, o in enumerate(((1, 1, 1), (0, 0, 1), (0, 1, 0), (1, 0, 0))):
        O.orc_calrn(*N, *inv, *[I(t) for t in o], *[P(a) for a in g], P(rn[q]))
    rk = np.zeros((3,) + sh)
    O.orc_calrkap(*N, *inv, *[P(r) for r in rn], P(rk))
    p = [np.zeros(sh) for _ in range(3)]
    O.orc_cal_grad_p2uvw(I(0), I(nj), *N, D(1 / dx), P(dya), D(1 / dz), P(phi), *[P(a) for a in p])
    ref = [np.zeros(sh) for _ in range(3)]
    O.orc_calfst(*N, D(rhol), D(rhog), D(sigma), *[P(a) for a in p], P(rk), *[P(a) for a in ref])
    got = _gpu(fmf_lib, ni, nj, nk, (dx, dy, dz), (rhol, rhog), sigma, phi)
    scale = 2 * sigma / (rhol + rhog) * max(1 / dx, 1 / dy, 1 / dz) ** 2
    for a, b in zip(got, ref):
        a, b = a[3:-3, 3:-3, 3:-3], b[3:-3, 3:-3, 3:-3]
        assert np.abs(b).max() > 0
        assert np.abs(a - b).max() <= 3e-14 * scale


def test_csf_fp64_nan_and_inf_are_not_flat(fmf_lib):
    """A NaN, and a field that is infinite everywhere, are not constant data."""
    ni, nj, nk = 64, 8, 16
    phi = np.ones((nk + 6, nj + 6, ni + 6))
    phi[10, 6, 40] = np.nan
    f = _gpu(fmf_lib, ni, nj, nk, (1.0, 1.0, 1.0), (1.0, 1.0), 1.0, phi)
    for a in f:
        assert np.isnan(a[10, 6, 40])
    f = _gpu(fmf_lib, ni, nj, nk, (1.0, 1.0, 1.0), (1.0, 1.0), 1.0, np.full(phi.shape, np.inf))
    for a in f:
        assert np.isnan(a[3:-3, 3:-3, 3:-3]).all()
