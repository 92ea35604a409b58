"""Every neighbour count around those at which a block's rows fill the shared memory that a kernel has without asking
(48 KB, its tables included), or at which it takes fewer rows: the perplexity search, the smooth-kNN search and the
transform's row search.

References: the oracle, with the tolerances of the tests of the whole graph and transform.
"""
import numpy as np
import pytest

import oracle as O
from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


def _knn(k):
    n = max(300, k + 5)
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    return idx, np.sort(np.random.default_rng(k).uniform(0.2, 3.0, (n, k)), 1).astype(np.float32)


@pytest.mark.parametrize("k", [45, 46, 47, 48, 94, 95, 96, 97, 110, 111, 112, 191, 192, 193, 222, 223, 224, 225])
def test_searches(k):
    idx, dist = _knn(k)
    perplexity = float(np.float32(k / 3))  # the library takes a float
    got = api.tsne_affinities(idx, dist, perplexity, index_offset=0)
    want, _ = O.row_p_f64(dist, perplexity)
    assert np.abs(got["p_directed"] - want).max() <= 2e-6 * want.max()
    graph = api.umap_graph(idx, dist, index_offset=0)
    offsets, neighbors, weights, _, _ = O.umap_graph(idx, dist, 0)
    np.testing.assert_array_equal(graph["offsets"], offsets)
    np.testing.assert_array_equal(graph["neighbors"], neighbors)
    np.testing.assert_allclose(graph["weights"], weights, rtol=2e-6)


@pytest.mark.parametrize("k", [255, 256, 257, 511, 512, 513])
def test_transform(k):
    rng = np.random.default_rng(k)
    ref = rng.normal(size=(2000, 2)) * 10
    idx = rng.integers(0, 2000, (40, k)).astype(np.int32)
    dist = np.sort(rng.uniform(0.2, 3.0, (40, k)), 1)
    got = api.transform_tsne(ref, dict(indices=idx, distances=dist), n_iter=5, perplexity=30.0)
    want = O.transform_tsne(ref, idx, dist, n_iter=5, perplexity=30.0)
    assert np.abs(got.layout - want).max() <= 1e-3
