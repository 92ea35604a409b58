"""PCA start of data with a column far from zero: the products are scaled by the centred data's magnitude, which such a
column does not raise.

Reference: FP64 with the same float centring. Tolerance as for other data: a score and the final product are each rounded
to float, half a unit in the last place of values up to the largest: 2^-23 of it in all, 2^-22 allowed.
"""
import numpy as np
import pytest

from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


def _start(x):
    mean = x.astype(np.float64).mean(0).astype(np.float32)
    xc = (x - mean).astype(np.float64)
    xc /= np.abs(xc).max()
    s = xc @ np.linalg.svd(xc, full_matrices=False)[2][:2].T
    s *= np.where(s[np.argmax(np.abs(s), 0), [0, 1]] < 0, -1.0, 1.0)
    s -= s.mean(0)
    return s * (1e-4 / s.std(0, ddof=1).max())


@pytest.mark.parametrize("constant", [0.0, 1e10, -1e15, 1e20, -1e23, 1e30, 3e38])
@pytest.mark.parametrize("n,p,scale", [(4096, 12, 1.0), (1025, 160, 1.0), (4096, 12, 1e-6)])
def test_constant_column(n, p, scale, constant):
    rng = np.random.default_rng(p)
    x = (rng.normal(size=(n, p)) * np.r_[3.0, 2.0, np.full(p - 2, 0.3)]) @ np.linalg.qr(rng.normal(size=(p, p)))[0]
    x = (x * scale).astype(np.float32)
    x[:, 1] = constant
    got, want = api.tsne_pca_init(x), _start(x)
    assert np.abs(got - want).max() <= 2.0 ** -22 * np.abs(want).max()
