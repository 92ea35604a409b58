"""Calls of different sizes on several threads. A kernel's limit of dynamic shared memory belongs to the process, so one
thread's launch must not depend on the size of another's; and no thread may wait for the device, or on the legacy stream,
while another captures its iterations in a graph. Every call's result is compared with its result alone, bit for bit."""
import threading

import numpy as np
import pytest

from fastembedr_gb300 import api

pytestmark = pytest.mark.gpu


def _spectral(n):
    i = np.arange(n)
    nb = np.sort(np.stack([(i - 1) % n, (i + 1) % n], 1), 1).astype(np.int32).ravel()
    graph = np.arange(0, 2 * n + 1, 2, dtype=np.int32), nb, np.ones(2 * n, np.float32)
    return lambda: api.umap_spectral_start_csr(*graph, 1, 3)


def _pca(p):
    x = np.random.default_rng(p).normal(size=(200, p)).astype(np.float32)
    return lambda: api.tsne_pca_init(x)


def _knn(k):
    n = 400
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    return idx, np.sort(np.random.default_rng(k).uniform(0.2, 3.0, (n, k)), 1).astype(np.float32)


def _affinities(k):
    idx, dist = _knn(k)
    return lambda: api.tsne_affinities(idx, dist, k / 3, index_offset=0)["p_directed"]


def _graph(k):
    idx, dist = _knn(k)
    return lambda: api.umap_graph(idx, dist, index_offset=0)["weights"]


def _tsne(n):
    k = 15
    idx = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.int32)
    rng = np.random.default_rng(n)
    dist = np.sort(rng.uniform(0.2, 3.0, (n, k)), 1).astype(np.float32)
    init = rng.normal(size=(n, 2)).astype(np.float32)
    return lambda: api.tsne_knn(idx, dist, perplexity=5.0, n_iter=5, early_exaggeration_iter=5, Y_init=init).layout


@pytest.mark.parametrize("make,large,small,reps", [(_spectral, 300000, (40, 100, 300, 900), 60), (_pca, 120, (3, 5, 9, 17), 120),
                                                   (_affinities, 100, (50, 55, 60, 70), 400),
                                                   (_graph, 100, (50, 55, 60, 70), 400),
                                                   (_tsne, 30000, (100, 300, 900, 2000), 60)])
def test_sizes_side_by_side(make, large, small, reps):
    faults, stop = [], threading.Event()

    def loop(f, want, count):
        while count != 0 and not (count < 0 and stop.is_set()):
            count -= 1
            try:
                if not np.array_equal(f(), want):
                    faults.append("differs")
            except Exception as e:  # noqa: BLE001
                faults.append(str(e))

    big, others = make(large), [make(k) for k in small for _ in range(2)]
    first, side = big(), [f() for f in others]
    runs = [threading.Thread(target=loop, args=(big, first, reps)) for _ in range(2)]
    back = [threading.Thread(target=loop, args=(f, w, -1)) for f, w in zip(others, side)]
    for t in runs + back:
        t.start()
    for t in runs:
        t.join()
    stop.set()
    for t in back:
        t.join()
    assert not faults, (len(faults), faults[0])
