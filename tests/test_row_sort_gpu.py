"""Row sorts of the t-SNE P and the UMAP fuzzy graph at the sizes where their path changes: rows of up
to 32, 64, 128 and 256 directed entries are sorted in a warp's registers, longer ones by a block.
Neighbours listed two, three and four times make runs that span lanes.

Structure is exact; values are held to the tolerance of the oracle's FP32 bisection (2e-6 mean relative)
for P and to 2e-6 for the fuzzy weights, as in the tests of the whole graph.
"""
import numpy as np
import pytest

import oracle as O
from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


def _knn(k, repeat):
    n = 420
    rng = np.random.default_rng(100 * k + repeat)
    idx = np.stack([rng.choice(n - 1, k, replace=False) for _ in range(n)])
    idx = (idx + (idx >= np.arange(n)[:, None])).astype(np.int32)
    if repeat > 1:  # every third row lists its first neighbour several times, and is listed by it
        m = min(repeat, k)
        idx[::3, :m] = idx[::3, :1]
        for i in range(0, n, 3):
            idx[idx[i, 0], : min(2, k)] = i
    dist = np.sort(rng.uniform(0.5, 3.0, (n, k)), 1).astype(np.float32)
    return idx, dist


@pytest.mark.parametrize("repeat", [1, 2, 4])
@pytest.mark.parametrize("k", [1, 8, 15, 16, 17, 31, 33, 48, 63, 65, 100, 129, 180])
def test_p_rows(k, repeat):
    idx, dist = _knn(k, repeat)
    perp = max(1.0, k / 3)
    a = api.tsne_affinities(idx, dist, perp, index_offset=0)
    rp, col, val, _ = O.csr_from_p(idx, O.row_p_f32(dist, perp), 0)
    np.testing.assert_array_equal(a["row_ptr"], rp)
    np.testing.assert_array_equal(a["col"], col)
    assert np.abs(a["val"] - val).sum() < 2e-6 * np.abs(val).sum()


@pytest.mark.parametrize("repeat", [1, 2, 4])
@pytest.mark.parametrize("k", [2, 8, 15, 16, 17, 31, 33, 63, 65, 100, 129, 180])
def test_fuzzy_rows(k, repeat):
    idx, dist = _knn(k, repeat)
    a = api.umap_graph(idx, dist, index_offset=0)
    offsets, neighbors, weights, _, _ = O.umap_graph(idx, dist, 0)
    np.testing.assert_array_equal(a["offsets"], offsets)
    np.testing.assert_array_equal(a["neighbors"], neighbors)
    assert np.abs(a["weights"] - weights).max() < 2e-6
    assert a["max_weight"] == np.max(a["weights"])
