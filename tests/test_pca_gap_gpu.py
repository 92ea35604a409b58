"""PCA start where the two leading eigenvalues differ by little: each eigenvector then takes up of the other what the
eigensolver leaves over the gap.

Reference: FP64 (SVD) with the same float centring. Tolerance: the products' two-float sums are good to about 2^-48 of
the largest eigenvalue and the refinement is FP64, so with a gap of 1e-7 the vectors mix by less than 2^-24; a score and
the final product are each rounded to float, half a unit in the last place of values up to the largest: 2^-22 of it
allowed in all. Feature counts on both sides of the largest matrix kept in shared memory (152), and the smallest.
"""
import numpy as np
import pytest

from fastembedr_gb300 import api
from test_pca_scale_gpu import _start

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gap", [1e-3, 1e-6, 1e-7])
@pytest.mark.parametrize("p", [2, 3, 50, 151, 152, 153, 200])
def test_close_eigenvalues(p, gap):
    n = 4000
    for seed in range(4):
        rng = np.random.default_rng(1000 * p + seed)
        u = rng.normal(size=(n, p))
        u = np.linalg.qr(u - u.mean(0))[0]
        s = np.r_[1.0, np.sqrt(1 - gap), np.linspace(0.9, 0.2, p - 2)]
        x = (100 * (u * s) @ np.linalg.qr(rng.normal(size=(p, p)))[0]).astype(np.float32)
        got, want = api.tsne_pca_init(x), _start(x)
        assert np.abs(got - want).max() <= 2.0 ** -22 * np.abs(want).max()
