"""KL divergence with the all-pairs normaliser at the edges of its 1024-point tiles, and its logarithm
over the whole range of P and q (nearly coincident to far apart points).

Reference: FP64 over the P that the library reports, with d^2 rounded to FP32 as the definition keeps it.
Tolerance: log(1 + d^2) of an FP32 d^2 is exact to 2^-24 relative of d^2, the normaliser is rounded to FP32
(2^-24) and its FP32 partial sums of 128 terms are within 2^-22: each moves the KL by less than 3e-7
absolute, and the KL of these inputs is above 0.3: 2e-6 relative.
"""
import numpy as np
import pytest

from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [1e-3, 3.0, 3e4])
@pytest.mark.parametrize("n", [4, 1023, 1024, 1025, 2049, 3000])
def test_kl_against_fp64(n, spread):
    rng = np.random.default_rng(n)
    k = min(6, n - 1)
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    dist = np.sort(rng.uniform(0.2, 4.0, (n, k)), 1).astype(np.float32)
    y = (rng.standard_normal((n, 2)) * spread).astype(np.float32)
    perp = max(1.0, k / 3)
    p = api.tsne_affinities(idx, dist, perp, index_offset=0)
    got = api.tsne_force_diagnostic(idx, dist, y, perp, 1.0, grid_size=32, exact=False, index_offset=0)["kl"]
    row = np.repeat(np.arange(n), np.diff(p["row_ptr"]))
    d = y[row] - y[p["col"]]
    d2 = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]).astype(np.float64)
    y64 = y.astype(np.float64)
    z = sum((1 / (1 + ((y64[s:s + 256, None] - y64[None]) ** 2).sum(2))).sum() for s in range(0, n, 256)) - n
    v = p["val"].astype(np.float64)
    want = (v * np.log((v + 1e-9) / (1 / (1 + d2) / max(z, 1e-38) + 1e-9))).sum()
    assert got == pytest.approx(want, rel=2e-6)
