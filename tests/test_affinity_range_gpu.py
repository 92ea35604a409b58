"""Perplexity search of rows whose precision leaves the float range (more neighbours tied at the smallest distance than
the perplexity, where the entropy never reaches the target and the precision is doubled 200 times), and of rows whose
squared distances nearly do.

Reference: the FP64 search of the oracle. Both take the same steps; a probability is rounded to float once: 2^-24 of
itself, 2^-23 allowed.
"""
import numpy as np
import pytest

import oracle as O
from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


def _ring(n, k):
    return ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)


@pytest.mark.parametrize("smallest", [0.0, 0.75])
@pytest.mark.parametrize("k,ties,perplexity", [(89, 50, 30.0), (6, 3, 2.0), (300, 200, 100.0)])
def test_more_ties_than_the_perplexity(k, ties, perplexity, smallest):
    n = 700
    rng = np.random.default_rng(k)
    dist = np.sort(smallest + rng.uniform(0.1, 3.0, (n, k)), 1).astype(np.float32)
    dist[::2, :ties] = smallest  # every other row; the others have no ties
    got = api.tsne_affinities(_ring(n, k), dist, perplexity, index_offset=0)
    want, beta = O.row_p_f64(dist, perplexity)
    assert beta[::2].min() > 3.4e38
    np.testing.assert_allclose(got["p_directed"][::2], want[::2], rtol=2.0 ** -23)
    np.testing.assert_allclose(got["entropy"][::2], np.log(ties), rtol=1e-12)
    assert np.isfinite(got["val"]).all() and np.isfinite(got["total_mass"])
    fit = api.tsne_knn(_ring(n, k), dist, perplexity=perplexity, n_iter=5, early_exaggeration_iter=5)
    assert np.isfinite(fit.layout).all()


# On both sides of 1e15, from where a row is searched in FP64, and up to 1.8e19, where a float's square overflows (such a
# row is uniform by the zero-spread test, which is in float as the reference's) and sums of several squares do before.
# Below the line the exponentials are FP32: an exponent x errs by 3 x 2^-24, which moves a probability p = exp(-x) / sum by
# less than 0.37 x 3 x 2^-24 of 1.
@pytest.mark.parametrize("lo,hi", [(2e14, 5e14), (8e14, 2e15), (1e18, 1.8e19)])
def test_squares_beyond_the_float_range(lo, hi):
    n, k = 500, 30
    rng = np.random.default_rng(7)
    dist = np.sort(rng.uniform(lo, hi, (n, k)), 1).astype(np.float32)
    got = api.tsne_affinities(_ring(n, k), dist, 10.0, index_offset=0)
    want, _ = O.row_p_f64(dist, 10.0)
    fp64 = dist.max(1) > 1.001e15
    np.testing.assert_allclose(got["p_directed"][fp64], want[fp64], rtol=2.0 ** -23)
    np.testing.assert_allclose(got["p_directed"][~fp64], want[~fp64], rtol=2.0 ** -22, atol=2.0 ** -23)
