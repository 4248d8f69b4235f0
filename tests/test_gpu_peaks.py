"""The measured pipe rates that the roofline fractions divide by: the FP64 GEMM
issues tensor instructions, whose rate is not that of FMA chains (37 and 34
TFLOP/s). A tenth is left for a clock that changes between the two launches."""
import ctypes

import pytest

from librascal_b200 import _native as N

pytestmark = pytest.mark.gpu


def test_rates():
    v = ctypes.c_double()
    N.check(N.lib().rgpu_measure_fp64_tensor_peak(ctypes.byref(v)))
    tensor = v.value
    N.check(N.lib().rgpu_measure_fma_peak(N.PRECISION_FP64, ctypes.byref(v)))
    fma64 = v.value
    N.check(N.lib().rgpu_measure_fma_peak(N.PRECISION_FP32, ctypes.byref(v)))
    assert 0 < 0.9 * fma64 < tensor < v.value
    assert N.lib().rgpu_measure_fp64_tensor_peak(None) == N.ERR_INVALID_ARGUMENT
