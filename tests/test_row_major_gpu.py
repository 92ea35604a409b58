"""Row-major and column-major host input give the same result (the library transposes row-major input on
the device, in 32 x 32 tiles), with 0- and 1-based labels of either integer width.

The transposes move values, so results are equal bit for bit, except UMAP's, whose asynchronous epochs
differ between identical runs: its fuzzy graph is compared through one epoch that samples nothing
(epoch 0), which returns the start.
"""
import numpy as np
import pytest

from fastembedr_gb300 import _lib, api

pytestmark = pytest.mark.gpu


def _knn(n, k, seed):
    rng = np.random.default_rng(seed)
    idx = np.stack([rng.choice(n - 1, k, replace=False) for _ in range(n)])
    idx = (idx + (idx >= np.arange(n)[:, None])).astype(np.int32)
    idx[1, 0], idx[0, 0] = 0, n - 1
    return idx, np.sort(rng.uniform(0.5, 3.0, (n, k)), 1).astype(np.float32)


@pytest.mark.parametrize("n,k", [(33, 1), (64, 31), (65, 32), (97, 33), (500, 65)])
def test_tsne_and_umap(n, k):
    idx, dist = _knn(n, k, n)
    y = np.random.default_rng(1).standard_normal((n, 2)).astype(np.float32)
    run = lambda i, d: api.tsne_knn(i, d, perplexity=max(1.0, k / 3), Y_init=y, early_exaggeration_iter=2, n_iter=2).layout
    want = run(np.asfortranarray(idx), np.asfortranarray(dist))
    for i in (idx, idx + 1, idx.astype(np.int64), (idx + 1).astype(np.int64), np.asfortranarray(idx + 1)):
        np.testing.assert_array_equal(run(i, dist), want)
    umap = lambda i, d: api.umap_knn(i, d, init=y, n_epochs=1).layout
    want = umap(np.asfortranarray(idx), np.asfortranarray(dist))
    for i in (idx, idx + 1):
        np.testing.assert_array_equal(umap(i, dist), want)


@pytest.mark.parametrize("nq,k", [(1, 1), (7, 33), (300, 20)])
def test_transform_and_server(nq, k):
    n_ref = 600
    rng = np.random.default_rng(nq)
    ref = rng.standard_normal((n_ref, 2)) * 5
    idx = rng.integers(0, n_ref, (nq, k)).astype(np.int32)
    idx[0, 0] = 0
    dist = np.sort(rng.uniform(0.5, 3.0, (nq, k)).astype(np.float32), 1)
    run = lambda i, d: api.transform_tsne(ref, dict(indices=i, distances=d), n_iter=5).layout
    want = run(np.asfortranarray(idx), np.asfortranarray(dist))
    np.testing.assert_array_equal(run(idx, dist), want)
    np.testing.assert_array_equal(run(idx + 1, dist), want)
    with api.TransformServer(ref, n_iter=5, memory_budget_bytes=1 << 28) as sv:
        ids = [sv.submit(idx, dist), sv.submit(np.asfortranarray(idx), np.asfortranarray(dist)), sv.submit(idx + 1, dist)]
        for r in ids:
            np.testing.assert_array_equal(sv.result(r)[0], want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n,p", [(33, 2), (100, 31), (257, 40)])
def test_pca(n, p, dtype):
    x = np.random.default_rng(p).standard_normal((n, p)).astype(dtype)
    np.testing.assert_array_equal(api.tsne_pca_init(x), api.tsne_pca_init(np.asfortranarray(x)))


def test_errors_are_those_of_column_major_input():
    idx, dist = _knn(50, 5, 3)
    for bad_idx, bad_dist in ((np.where(idx == idx[4, 2], 51, idx).astype(np.int32), dist), (idx, -dist),
                              (idx, np.where(dist == dist[3, 1], np.nan, dist).astype(np.float32))):
        said = []
        for order in (np.ascontiguousarray, np.asfortranarray):
            with pytest.raises(_lib.CudaEmbeddingError) as e:
                api.tsne_knn(order(bad_idx), order(bad_dist), perplexity=2.0, n_iter=1, early_exaggeration_iter=0)
            said.append(str(e.value))
        assert said[0] == said[1]
