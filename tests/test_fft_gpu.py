"""Grid repulsion at every transform length (G = 8 .. 1024 nodes, M = 2 G) and both stencils.

Each length has its own passes in registers, its own shared-memory order and, below 128 nodes, several
sequences per warp; the Lagrange stencil uses 3 floor(G / 3) nodes, odd for some G, which leaves the
last row pair half empty. Reference: the same interpolation scheme in FP64.

Tolerance: a value passes 4 log2(M) butterflies of about 2 roundings (2^-24 each, adding up as a random
walk: sqrt(8 x 11) x 6e-8 = 6e-7) and the force is a difference of terms up to about ten times its size;
1e-5 relative L2 leaves a factor of two.
"""
import numpy as np
import pytest

import oracle as O
from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("grid", [8, 16, 32, 64, 128, 256, 512, 1024])
def test_every_transform_length(grid, mode):
    n, k = 1500, 5
    rng = np.random.default_rng(grid + mode)
    y = (rng.standard_normal((n, 2)) * [4.0, 2.5] + [1.0, -3.0]).astype(np.float32)
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    dist = np.sort(rng.uniform(0.5, 2.0, (n, k)), 1).astype(np.float32)
    got = api.tsne_force_diagnostic(idx, dist, y, 1.5, 1.0, grid_size=grid, interpolation=mode, exact=False, kl=False)
    want, z = O.interp_rep_f64(y, grid, lagrange=mode)
    assert got["z_grid"] == pytest.approx(z, rel=1e-5)
    assert np.linalg.norm(got["repulsive_force_fft"] - want) < 1e-5 * np.linalg.norm(want)
