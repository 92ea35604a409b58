"""KL divergence of layouts so wide that every q is small: q / Z is of the order of 1 / n^2 all the same.

Reference: FP64 over the P that the library reports, with d^2 rounded to FP32 as the definition keeps it; Z without the
pairs (i, i). Tolerance: 2e-6, as for other layouts (test_kl_gpu).
"""
import numpy as np
import pytest

from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [1e12, 3e14, 3e15, 1e18])
def test_kl_of_wide_layouts(spread):
    n, k = 1500, 6
    rng = np.random.default_rng(5)
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    dist = np.sort(rng.uniform(0.2, 4.0, (n, k)), 1).astype(np.float32)
    y = (rng.standard_normal((n, 2)) * spread).astype(np.float32)
    p = api.tsne_affinities(idx, dist, 2.0, index_offset=0)
    got = api.tsne_force_diagnostic(idx, dist, y, 2.0, 1.0, grid_size=32, exact=False, index_offset=0)["kl"]
    row = np.repeat(np.arange(n), np.diff(p["row_ptr"]))
    d = y[row] - y[p["col"]]
    q = 1 / (1 + (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).astype(np.float64))
    y64 = y.astype(np.float64)
    pairs = 1 / (1 + ((y64[:, None] - y64[None]) ** 2).sum(2))
    np.fill_diagonal(pairs, 0.0)
    v = p["val"].astype(np.float64)
    want = (v * np.log((v + 1e-9) / (q / pairs.sum() + 1e-9))).sum()
    assert got == pytest.approx(want, rel=2e-6)
