"""Perplexity search of rows whose precision leaves the float range: more neighbours tied at the smallest distance than
the perplexity, where the entropy never reaches the target and the precision is doubled 200 times.

Reference: the FP64 search of the oracle. Both end at the same precision, far beyond the float range, where the tied
neighbours share the mass and the others have none; a probability is rounded to float once: 2^-24 of itself, 2^-23
allowed.
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
