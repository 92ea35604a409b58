"""UMAP's curve parameters fitted beside a job (the grid of least squares on the GPU) are those of the host function,
bit for bit. (Against the oracle they agree to 1e-9 up to min_dist 0.9; beyond, the descent amplifies the compiler's
choice of fused multiply-adds.)"""
import ctypes as C

import numpy as np
import pytest

from fastembedr_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("min_dist", [*np.round(np.arange(0.0, 1.05, 0.045), 3), 0.001, 0.01, 0.1, 0.25, 0.5, 0.99, 2.5, 100.0,
                                      float(np.float32(0.01)), float(np.float32(0.1)), float("nan"), float("inf")])
def test_curve_is_the_host_function_bit_for_bit(min_dist):
    a, b, ra, rb = C.c_double(), C.c_double(), C.c_double(), C.c_double()
    lib = _lib.require_gpu()
    _lib.check(lib.fastembedr_cuda_umap_find_ab_params(1.0, min_dist, C.byref(a), C.byref(b)), "curve")
    lib.fastembedr_umap_find_ab_params(1.0, min_dist, C.byref(ra), C.byref(rb))
    assert (a.value, b.value) == (ra.value, rb.value)
