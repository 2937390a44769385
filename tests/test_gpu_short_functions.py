"""The third-order reciprocal and reciprocal square root (csrc/recip.cuh) and the interface
band's short exponential, which the FP64 kernels call, against the functions they stand for."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name, ulps", [("fmf_check_reciprocal", 2), ("fmf_check_rsqrt", 2),
                                        ("fmf_check_exponential", 3)])
@pytest.mark.parametrize("n", [1 << 16, (1 << 24) + 1])
def test_error(fmf_lib, name, ulps, n):
    """In units of 2^-52.  Reciprocals: a half each for the result's last rounding and the
    comparison's, a little for the step's.  Exponential: one each for the tabulated value and
    exp, a half for the last rounding, 0.1 for the polynomial's sum."""
    fn = getattr(fmf_lib, name)
    fn.argtypes = [ctypes.c_longlong, ctypes.POINTER(ctypes.c_double)]
    err = ctypes.c_double(-1.0)
    assert fn(n, ctypes.byref(err)) == 0
    assert 0.0 < err.value <= ulps * 2.0 ** -52, err.value
    assert fn(0, ctypes.byref(err)) == 2 and fn(n, None) == 2  # FMF_ERR_ARG
