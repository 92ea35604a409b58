"""The spectral start's normal draws made on the GPU against the host's stream: the same words, accepted points and order, so
that every draw differs by the rounding of its logarithm only.

Tolerance: CUDA's and the host's logarithm are each within a unit in the last place; root, quotient and four products
behind them round each side once more: 8 units in all, 2^-50 of a draw.
"""
import ctypes as C

import numpy as np
import pytest

from fastembedr_gb300 import _lib

pytestmark = pytest.mark.gpu


def _draws(seed, count, max_points=0):
    dev, host, enough = np.zeros(count), np.zeros(count), C.c_int(-1)
    st = _lib.require_gpu().fastembedr_cuda_normal_draws(seed, count, max_points, dev.ctypes.data, host.ctypes.data,
                                                         C.byref(enough))
    _lib.check(st, "normal draws")
    return dev, host, enough.value


@pytest.mark.parametrize("seed", [0, 1, 42, 4294967295])
@pytest.mark.parametrize("count", [2, 8190, 65536, 65538, 1600000])
def test_draws_follow_the_host_stream(seed, count):
    dev, host, enough = _draws(seed, count)
    assert enough == 1
    np.testing.assert_allclose(dev, host, rtol=2.0 ** -50)


def test_too_few_words_are_reported():
    dev, _, enough = _draws(3, 65536, max_points=32768)  # a point in five is rejected
    assert enough == 0 and not dev.any()
