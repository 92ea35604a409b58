"""Scatter of the charges where points lie beyond their block's tile: counts of such points in a warp from one to 32 (the
last warp ragged), all in the tile, all beyond it, and both stencils."""
import numpy as np
import pytest

from fastembedr_gb300 import api
import oracle as O

pytestmark = pytest.mark.gpu


# A point's repulsion is (y phi_q2 - phi_xy) / Z: terms of size |y - c| phi_q2, its own charge included, cancel down to it
# (for a few points far apart by three digits). The potentials carry the rounding of a forward and an inverse
# transform in two dimensions, 4 log2 M <= 36 butterfly levels of 6e-8, and the Lagrange weights add up to 2.44 in
# magnitude: 5.4e-6 of those terms. The same interpolation in FP64 is the oracle.
@pytest.mark.parametrize("n,grid,spread", [(9, 256, 1.0), (31, 256, 1.0), (33, 256, 1.0), (257, 256, 1.0), (300, 64, 1.0),
                                           (700, 256, 0.02)])
@pytest.mark.parametrize("lagrange", [0, 1])
def test_charges_of_spread_and_of_compact_layouts(n, grid, spread, lagrange):
    rng = np.random.default_rng(n + grid)
    k = 3
    idx = (np.arange(n)[:, None] + 1 + np.arange(k)[None, :]) % n
    dist = np.sort(rng.uniform(0.5, 2.0, (n, k)), 1).astype(np.float32)
    y = (rng.uniform(-10.0, 10.0, (n, 2)) * spread).astype(np.float32)
    y[: min(4, n)] = [[-10, -10], [10, 10], [-10, 10], [10, -10]][: min(4, n)]  # the box, whatever the spread
    d = api.tsne_force_diagnostic(idx.astype(np.int32), dist, y, 1.0, grid_size=grid, interpolation=lagrange, exact=False,
                                  kl=False, index_offset=0)
    want, z = O.interp_rep_f64(y, grid, lagrange)
    x = y.astype(np.float64)
    phi = ((1.0 / (1.0 + ((x[:, None] - x[None]) ** 2).sum(2))) ** 2).sum(1)
    terms = np.linalg.norm(x - 0.5 * (x.min(0) + x.max(0)), axis=1) * phi
    assert np.linalg.norm(d["repulsive_force_fft"] * d["z_grid"] - want * z) < 5.4e-6 * np.linalg.norm(terms)
