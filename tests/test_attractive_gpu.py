"""The attractive pass at the edges of its schedule and of a row's rounds.

The launch gives every warp one chunk of up to 8 rows, or feeds the warps from one queue per SM; a
row is read in rounds of 128 entries and a last round of 64 or 32. Reference: the same sums in
FP64 over the P that the library reports.

Tolerance: a term has about 8 FP32 roundings (two differences, d^2, reciprocal, two products) and a
row's sum 10 more (at most 4 entries a lane and round, 5 butterfly levels, Kahan between rounds), each
2^-24 of the partial sums, which exceed the row's result by the cancellation of its terms (here about
sqrt(entries) < 16 in the norm): 18 x 6e-8 x 4 < 5e-6 relative L2.
"""
import numpy as np
import pytest

from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


def _check(idx, dist, seed):
    n = idx.shape[0]
    y = (np.random.default_rng(seed).standard_normal((n, 2)) * 3.0).astype(np.float32)
    perp = max(1.0, idx.shape[1] / 3)
    p = api.tsne_affinities(idx, dist, perp, index_offset=0)
    got = api.tsne_force_diagnostic(idx, dist, y, perp, 4.0, grid_size=32, exact=False, kl=False, index_offset=0)
    row = np.repeat(np.arange(n), np.diff(p["row_ptr"]))
    d = y[row].astype(np.float64) - y[p["col"]]
    c = 4.0 * p["val"].astype(np.float64) / (1.0 + (d * d).sum(1))
    want = np.stack([np.bincount(row, c * d[:, a], n) for a in (0, 1)], 1)
    assert np.linalg.norm(got["attractive_force"] - want) < 5e-6 * np.linalg.norm(want)
    return np.diff(p["row_ptr"])


# around one row a warp, the largest static chunk (8 rows for each of 152 x 48 warps), the queues
@pytest.mark.parametrize("n", [2, 31, 7296, 7297, 58_367, 58_368, 58_369, 200_003])
def test_every_schedule_takes_every_row(n):
    rng = np.random.default_rng(n)
    k = min(4, n - 1)
    idx = ((np.arange(n)[:, None] + 1 + rng.integers(0, max(1, n - k), (n, 1)) % max(1, n - k)
            + np.arange(k)[None, :]) % n).astype(np.int32)
    idx = np.where(idx == np.arange(n)[:, None], (idx + 1) % n, idx).astype(np.int32)
    dist = np.sort(rng.uniform(0.5, 2.0, (n, k)), 1).astype(np.float32)
    _check(idx, dist, n)


@pytest.mark.parametrize("k", [1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200])
def test_row_lengths_around_the_rounds(k):
    """Hubs and leaves: rows of k to several hundred entries, starting at every position modulo 4."""
    n = 700
    rng = np.random.default_rng(k)
    idx = np.stack([rng.choice(n - 1, k, replace=False) for _ in range(n)])
    idx = (idx + (idx >= np.arange(n)[:, None])).astype(np.int32)
    idx[:, 0] = np.where(np.arange(n) == 5, idx[:, 0], 5)
    dist = np.sort(rng.uniform(0.5, 2.0, (n, k)), 1).astype(np.float32)
    rows = _check(idx, dist, k)
    assert rows[5] >= n // 2
