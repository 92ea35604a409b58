"""Transform queries at the sizes where a path changes: neighbours in registers (up to 128), rows cached in
shared memory (median: up to 256, search: up to 512), one to eight warps a block, and reference coordinates
that tie, are negative or signed zeros in the median.

Reference: the FP64 oracle of transform_tsne. Tolerance: the tests of the whole transform hold 250
iterations to 1e-3 (median) and 1e-2 (99 %); three iterations of FP32 forces on steps of at most 0.25
a component move a point by less than 1.5, so 18 FP32 roundings a step give 3 x 18 x 6e-8 x 1.5 < 1e-5.
"""
import numpy as np
import pytest

import oracle as O
from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("init", ["median", "weighted"])
@pytest.mark.parametrize("k", [1, 2, 31, 32, 33, 127, 128, 129, 256, 257, 512, 513])
def test_row_lengths(k, init):
    n_ref, nq = 900, 21
    rng = np.random.default_rng(k)
    ref = np.round(rng.standard_normal((n_ref, 2)) * 8) / 4  # many ties
    ref[::7] = 0.0
    ref[::14] = -0.0
    idx = np.stack([rng.choice(n_ref, k, replace=False) for _ in range(nq)]).astype(np.int32)
    idx[0, 0] = 0
    dist = np.sort(rng.uniform(0.5, 3.0, (nq, k)), 1)
    got = api.transform_tsne(ref, dict(indices=idx, distances=dist), n_iter=3, perplexity=max(1.0, min(5.0, k / 3)),
                             initialization=init, seed=3).layout
    want = O.transform_tsne(ref, idx, dist, n_iter=3, perplexity=max(1.0, min(5.0, k / 3)), n_negatives=900,
                            exact_threshold=4096, init_mode=1 if init == "median" else 2, seed=3)
    assert np.abs(got - want).max() < 1e-5


@pytest.mark.parametrize("nq", [1, 151, 153, 305, 1217])
def test_query_counts(nq):
    n_ref, k = 400, 12
    rng = np.random.default_rng(nq)
    ref = rng.standard_normal((n_ref, 2)) * 5
    idx = rng.integers(0, n_ref, (nq, k)).astype(np.int32)
    idx[0, 0] = 0
    dist = np.sort(rng.uniform(0.5, 3.0, (nq, k)), 1)
    got = api.transform_tsne(ref, dict(indices=idx, distances=dist), n_iter=3, seed=3).layout
    want = O.transform_tsne(ref, idx, dist, n_iter=3, n_negatives=400, exact_threshold=4096, seed=3)
    assert np.abs(got - want).max() < 1e-5
