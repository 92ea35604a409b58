"""The subspace iteration of the CPU spectral start at the edges of its row split: fewer rows than a warp, one and two
warps per block (152 blocks of 32 rows hold 4,864), one and two tiles (77,824 rows), rows in the global buffers (more
than 524,552), fewer points than the block has columns, and both sides of the line (8,192) from which the start
block is drawn on the GPU."""
import numpy as np
import pytest

from fastembedr_gb300 import api
import oracle as O

pytestmark = pytest.mark.gpu


def ring(n, rng):
    """A symmetric CSR graph: a ring of random weights."""
    w = rng.uniform(0.2, 1.0, n).astype(np.float32)  # w[i] joins i and i + 1
    i = np.arange(n)
    nb = np.stack([(i - 1) % n, (i + 1) % n], 1).astype(np.int32)
    wt = np.stack([np.roll(w, 1), w], 1)
    order = np.argsort(nb, 1)
    return (np.arange(0, 2 * n + 1, 2, dtype=np.int32), np.take_along_axis(nb, order, 1).ravel(),
            np.take_along_axis(wt, order, 1).ravel())


# Same operations as the oracle but for the order of the FP64 sums over points. A Ritz vector moves by the rounding of
# the projected matrix (1e-16 sqrt(n) at most) over the gap of the Ritz values, which for 8 random directions is
# above 1e-4 but for rare draws: 1e-9 of the layout's 10, and four decades of room for the division by the largest
# coordinate and the rounds' own amplification.
@pytest.mark.parametrize("n,iters", [(5, 3), (31, 3), (33, 3), (4864, 3), (4865, 3), (8191, 3), (8192, 3), (30001, 2), (77824, 2), (77825, 2), (100001, 2),
                                     (560000, 1)])
def test_spectral_rounds_edges(n, iters):
    off, nb, w = ring(n, np.random.default_rng(n))
    got = api.umap_spectral_start_csr(off, nb, w, iters, 3)
    want = O.umap_spectral_init(off, nb, w, iters, 3)
    assert np.abs(got - want).max() <= 1e-4, np.abs(got - want).max()
