"""Relabelling of P's columns at every reorder, by rows in storage order: fewer rows than blocks, rows starting at every
position modulo 4, empty shares of the last blocks, hub rows of several rounds of 128 entries."""
import numpy as np
import pytest

from fastembedr_gb300 import api
import oracle as O

pytestmark = pytest.mark.gpu


# The divergence of the layout under the relabelled P against the oracle's on the layout alone: a wrong label moves it in
# the first digits; both sum in FP64 or the like over terms of FP32 probabilities (relative 6e-8 each), 1e-5 allowed.
@pytest.mark.parametrize("n,k", [(7, 3), (33, 5), (300, 31), (1001, 129), (5003, 10), (20011, 17)])
def test_every_column_follows_its_point(n, k):
    import torch

    rng = np.random.default_rng(n)
    idx = np.stack([rng.choice(n - 1, k, replace=False) for _ in range(n)])
    idx = (idx + (idx >= np.arange(n)[:, None])).astype(np.int32)
    for row in range(n):  # point 5 is everybody's neighbour
        if row != 5 and 5 not in idx[row]:
            idx[row, 0] = 5
    dist = np.sort(rng.uniform(0.5, 2.0, (n, k)), 1).astype(np.float32)
    perp = max(1.0, k / 3)
    init = (rng.standard_normal((n, 2)) * 3).astype(np.float32)
    plan = api.TsnePlan(torch.as_tensor(np.ascontiguousarray(idx.T), device="cuda"),
                        torch.as_tensor(np.ascontiguousarray(dist.T), device="cuda"), n, k, perp, init=init)
    rp, col, val, _ = O.tsne_csr(idx, dist, perp)
    for _ in range(3):  # every run starts with a reorder
        plan.run(2, 1.0, n / 12.0)
        assert plan.kl() == pytest.approx(O.kl(rp, col, val, plan.layout()), rel=1e-5)
    plan.close()
