"""What a handle prepares before it launches anything."""
import ctypes

import pytest

import dgpr_b200 as dg


@pytest.mark.parametrize("curved", [0, 1])
@pytest.mark.parametrize("precision", [dg.FP64, dg.MIXED_FP32])
@pytest.mark.parametrize("p", [0, 1, 2, 3])
def test_no_kernel_is_loaded_ahead(p, precision, curved):
    """Setting a kernel's shared-memory limit loads it.  Up to p = 3 every
    kernel needs at most the 48 KB that it may have anyway, so preparing a
    handle and its adjoint makes no CUDA call, and passes without a GPU."""
    fn = dg.lib().dgb_check_prepare
    fn.restype, fn.argtypes = ctypes.c_int, [ctypes.c_int] * 3
    assert fn(p, precision, curved) == dg.OK
