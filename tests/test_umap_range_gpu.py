"""Fuzzy graph of distances whose sums leave the float range: a row's bandwidth is at least 1e-3 of its mean distance,
which is then all that keeps its weights above zero (the search doubles the bandwidth 64 times at most).

Reference: the oracle. Weights to 2e-6, as in the tests of the whole graph.
"""
import numpy as np
import pytest

import oracle as O
from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e36, 3e37, 3e38])
@pytest.mark.parametrize("k", [5, 15, 40])
def test_large_distances(k, scale):
    n = 300
    rng = np.random.default_rng(k)
    idx = np.stack([rng.choice(n - 1, k, replace=False) for _ in range(n)])
    idx = (idx + (idx >= np.arange(n)[:, None])).astype(np.int32)
    dist = (np.sort(rng.uniform(0.995, 1.0, (n, k)), 1) * scale).astype(np.float32)
    got = api.umap_graph(idx, dist, index_offset=0)
    offsets, neighbors, weights, _, _ = O.umap_graph(idx, dist, 0)
    np.testing.assert_array_equal(got["offsets"], offsets)
    np.testing.assert_array_equal(got["neighbors"], neighbors)
    np.testing.assert_allclose(got["weights"], weights, rtol=2e-6)
