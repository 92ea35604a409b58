"""PCA start on the device at the edges of its kernels: odd and even feature counts, feature counts beside the
Gram tile (16) and on both sides of the largest matrix the eigensolver keeps in shared memory (152), row counts beside
the 64-row chunks and the 1,024-row slices, and data whose squares leave the float range."""
import numpy as np
import pytest

from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


def pca_start(x):
    """FP64 restatement: float32 centring, eigenvectors by the SVD of the centred data, scores with the entry of
    largest magnitude positive, scaled by 1e-4 over the larger standard deviation."""
    xf = np.asarray(x, np.float32)
    mean = xf.astype(np.float64).mean(0).astype(np.float32)
    xc = (xf - mean).astype(np.float64)
    xc = xc / np.abs(xc).max()
    s = xc @ np.linalg.svd(xc, full_matrices=False)[2][:2].T
    for c in range(2):
        if s[np.argmax(np.abs(s[:, c])), c] < 0:
            s[:, c] = -s[:, c]
    s = s - s.mean(0)
    return s * (1e-4 / s.std(0, ddof=1).max())


# Column spreads fall by at least 8% from one to the next for the two leading components (3, 2, then 1), so
# eigenvectors are separated by eigenvalue gaps above a third of the spectrum: errors of the two-float sums
# (2^-40) do not show, and what is left is the rounding of a score to float and the final product, each half
# a unit in the last place of values up to the largest: 2^-23 of it in all, 2^-22 allowed.
@pytest.mark.parametrize("n,p,scale", [(3, 2, 1.0), (63, 3, 1.0), (64, 15, 1.0), (65, 16, 1.0), (1023, 17, 1.0),
                                       (1025, 33, 1.0), (5000, 151, 1.0), (5000, 152, 1.0), (5000, 153, 1.0),
                                       (3000, 260, 1.0), (70001, 50, 1.0), (4000, 20, 1e30), (4000, 20, 1e-30)])
def test_pca_start_edges(n, p, scale):
    rng = np.random.default_rng(n + p)
    z = rng.normal(size=(n, p))
    z[:, 2:] *= 0.3
    z[:, 0] *= 3.0
    z[:, 1] *= 2.0
    q = np.linalg.qr(rng.normal(size=(p, p)))[0]
    x = ((z @ q + rng.normal(size=p)) * scale).astype(np.float32)
    got = api.tsne_pca_init(x)
    want = pca_start(x)
    assert np.abs(got - want).max() <= 2.0 ** -22 * np.abs(want).max()


def test_constant_columns_give_zero_scores():
    x = np.tile(np.arange(5, dtype=np.float32), (100, 1))
    np.testing.assert_array_equal(api.tsne_pca_init(x), np.zeros((100, 2), np.float32))


def test_values_at_the_float_limit():
    """Column sums and squares beyond the float range: the means are 1e38 and the scores finite."""
    x = np.full((4096, 3), 1e38, np.float32)
    x[::2, 0] = 2e38
    x[1::2, 0] = 0.0
    x[::8, 1] = 1.2e38
    got = api.tsne_pca_init(x)
    want = pca_start(x)
    assert np.abs(got - want).max() <= 2.0 ** -22 * np.abs(want).max()
