"""The subspace iteration of the CPU spectral start on fewer SMs than it has partial slots for (152): one block, a few, and
148, with rows in shared memory (up to 3,456 a block) and in the global buffers, on one and on several tiles of 512 rows.

Reference: the oracle. Only the order of FP64 sums over points differs from the run on all SMs, so the bound is that of
test_spectral_rounds_gpu: 1e-4 of a layout of 10.
"""
import numpy as np
import pytest

from fastembedr_gb300 import _lib
import oracle as O
from test_spectral_rounds_gpu import ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,blocks", [(5, 1), (33, 1), (3456, 1), (3457, 1), (4865, 3), (10369, 3), (4737, 148),
                                      (20000, 148), (75777, 148)])
def test_fewer_blocks(n, blocks):
    off, nb, w = ring(n, np.random.default_rng(n))
    out = np.zeros(2 * n)
    st = _lib.require_gpu().fastembedr_cuda_umap_spectral_init_csr_blocks(
        off.ctypes.data, nb.ctypes.data, w.ctypes.data, n, 3, float("nan"), 3, blocks, out.ctypes.data)
    _lib.check(st, "CUDA spectral start")
    want = O.umap_spectral_init(off, nb, w, 3, 3)
    assert np.abs(out.reshape(2, n).T - want).max() <= 1e-4
