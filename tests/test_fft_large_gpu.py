"""Grid repulsion at the largest transform length that is accepted (G = 2048 nodes, M = 4096) and both stencils.

Reference and tolerance as for the other lengths (test_fft_gpu): the interpolation scheme in FP64, 1e-5 relative L2 for
48 butterflies a value.
"""
import pytest

from test_fft_gpu import test_every_transform_length as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
def test_largest_transform(mode):
    check(2048, mode)
