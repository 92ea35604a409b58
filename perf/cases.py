"""Performance cases of the embedding optimizer, driven through its public Python entry points.

Inputs are Gaussian mixtures with a decaying spectrum (what PCA scores of real data look like) and
well separated clusters, so the exact neighbours of a point lie in its own cluster and the KNN graph
of a million points is built in about a second. The kinds of work:

* ``plan``: iterations of a resident t-SNE instance (``TsnePlan.run`` + ``layout``), in the normal
  phase from a spread layout or in early exaggeration from a compact one;
* ``fit_device`` / ``fit_host``: a fit from the KNN graph (affinities, symmetrised P, iterations,
  layout) from device tensors or host arrays, cut to a few iterations of each phase;
* ``batch``: iterations of many uneven instances at once;
* ``umap`` / ``umap_spectral``: ``umap_knn`` from a given start, or from its default spectral start;
* ``pca``: the PCA start of t-SNE; ``kl``: the KL divergence of a fit;
* ``transform``: one ``transform_tsne`` call; ``serve``: a burst of requests to the transform server.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fastembedr_gb300 import api

DIM = 50

# Learning rates of a layout that is refined from a start the user has: t-SNE's default is n / 12 and
# UMAP's 1. The work of an iteration does not depend on them; at the defaults the first iterations
# from such a start amplify a rounding difference until two correct runs no longer agree.
TSNE_RATE = 1.0 / 120.0
UMAP_RATE = 0.1
SPECTRAL_RATE = 0.02


def listed():
    return [
        # the smallest resident fit: every kernel is short, launches and their latency count
        dict(name="tsne_2k", kind="plan", n=2000, k=90, early=False, iters=20),
        # a mid-size data set in the first phase: clusters collapsed onto few grid cells
        dict(name="tsne_200k_early", kind="plan", n=200_000, k=90, early=True, iters=10),
        # the headline: one million points in the normal phase
        dict(name="tsne_1m", kind="plan", n=1_000_000, k=90, early=False, iters=20),
        # tsne_knn() on host matrices, the plain 10k workload, first iterations of both phases
        dict(name="tsne_knn_10k", kind="fit_host", n=10_000, k=90, early_iters=5, iters=10),
        # a fit from a device KNN graph at an odd size and a short neighbour list: affinities dominate
        dict(name="tsne_fit_100k", kind="fit_device", n=100_003, k=45, early_iters=5, iters=5),
        # many uneven data sets optimised together
        dict(name="tsne_batch", kind="batch", instances=32, lo=2000, hi=20_000, k=90, sizes=7, iters=10),
        # umap_knn() from a start the user has: graph build and epochs
        dict(name="umap_100k", kind="umap", n=100_000, k=15, epochs=20),
        # umap_knn() as called by default: graph, spectral start, epochs; an odd size
        dict(name="umap_spectral_20k", kind="umap_spectral", n=20_003, k=15, epochs=10),
        # PCA start of t-SNE on a mid-size data matrix
        dict(name="pca_200k", kind="pca", n=200_000, p=50, double=False),
        # a serving burst: mixed request sizes into a large reference layout (sampled repulsion)
        dict(name="serve_burst", kind="serve", n_ref=200_000, requests=12, lo=1, hi=8000, k=90, sizes=11),
        # one small transform call (exact repulsion against a small reference), latency
        dict(name="transform_300", kind="transform", n_ref=2000, n_query=300, k=15, weighted=False),
        # KL divergence of a fit, all-pairs normaliser
        dict(name="kl_100k", kind="kl", n=100_000, k=30),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "plan", "fit_host", "fit_device", "batch", "umap", "umap", "umap_spectral",
                       "pca", "serve", "transform", "kl"])
    if kind == "plan":
        early = rng.random() < 0.4
        return dict(kind=kind, n=_log_int(rng, 1000, 1_000_000), k=rng.randint(15, 90), early=early,
                    iters=rng.randint(5, 10) if early else rng.randint(10, 20))
    if kind == "fit_host":
        return dict(kind=kind, n=_log_int(rng, 1000, 20_000), k=rng.randint(15, 90), early_iters=rng.randint(3, 5),
                    iters=rng.randint(3, 10))
    if kind == "fit_device":
        return dict(kind=kind, n=_log_int(rng, 2000, 200_000), k=rng.randint(15, 90), early_iters=5, iters=5)
    if kind == "batch":
        return dict(kind=kind, instances=rng.randint(2, 40), lo=1000, hi=_log_int(rng, 4000, 24_000),
                    k=rng.randint(15, 90), sizes=rng.randint(0, 10**6), iters=10)
    if kind == "umap":
        return dict(kind=kind, n=_log_int(rng, 1000, 200_000), k=rng.randint(5, 30), epochs=rng.randint(10, 25))
    if kind == "umap_spectral":
        return dict(kind=kind, n=_log_int(rng, 3000, 30_000), k=rng.randint(10, 20), epochs=rng.randint(5, 10))
    if kind == "pca":
        return dict(kind=kind, n=_log_int(rng, 1000, 200_000), p=rng.randint(5, 100), double=rng.random() < 0.5)
    if kind == "serve":
        return dict(kind=kind, n_ref=_log_int(rng, 20_000, 200_000), requests=rng.randint(3, 16), lo=1,
                    hi=_log_int(rng, 500, 8000), k=rng.randint(10, 90), sizes=rng.randint(0, 10**6))
    if kind == "transform":
        n_ref = _log_int(rng, 300, 4000)
        return dict(kind=kind, n_ref=n_ref, n_query=_log_int(rng, 1, 2000), k=rng.randint(3, 40),
                    weighted=rng.random() < 0.5)
    return dict(kind=kind, n=_log_int(rng, 2000, 100_000), k=rng.randint(15, 90))


# ---------------------------------------------------------------------------- inputs
def _clusters(n, gen, k):
    """Cluster sizes of a log-normal mixture, each larger than k + 1."""
    m = max(1, min(40, n // 500, n // (4 * (k + 1))))
    w = torch.exp(0.6 * torch.randn(m, generator=gen)).double().numpy()
    floor = 2 * (k + 1) if m > 1 else 0
    size = np.floor(w / w.sum() * (n - floor * m)).astype(np.int64) + floor
    size[0] += n - size.sum()
    return size


def _mixture(n, seed, k, extra=0):
    """Rows of the mixture in random order: data (n + extra, DIM) on the GPU, a 2-D layout like a
    fitted one (each cluster a disc whose area follows its size), and the rows of each cluster."""
    gen = torch.Generator().manual_seed(int(seed))
    g = torch.Generator("cuda").manual_seed(int(seed))
    size = _clusters(n + extra, gen, k)
    m = len(size)
    lab = torch.repeat_interleave(torch.arange(m), torch.from_numpy(size)).cuda()
    lab = lab[torch.randperm(n + extra, generator=g, device="cuda")]
    centre = 4.0 * torch.randn(m, DIM, generator=gen).cuda()
    z = torch.randn(n + extra, DIM, generator=g, device="cuda")
    sd = 3.0 / torch.sqrt(torch.arange(1, DIM + 1, device="cuda", dtype=torch.float32))
    x = centre[lab] + z * sd
    # discs on a spiral, sized by the cluster, over a span of about 100
    frac = torch.from_numpy(size / size.sum())
    ang = 2.399963 * torch.arange(m)
    mid = 45.0 * torch.sqrt((torch.arange(m) + 0.5) / m)
    at = torch.stack([mid * torch.cos(ang), mid * torch.sin(ang)], 1) if m > 1 else torch.zeros(1, 2)
    rad = 45.0 * torch.sqrt(frac).float()
    r2 = (z[:, :2] ** 2).sum(1, keepdim=True)
    y = at.float().cuda()[lab] + rad.cuda()[lab][:, None] * z[:, :2] * torch.sqrt((1 - torch.exp(-r2 / 2)) / r2)
    rows = [torch.nonzero(lab == c).ravel() for c in range(m)]
    return x, y, rows


def _search(q, r, k, self_rows):
    """Exact KNN of the rows q among the rows r (float32 distances, ascending)."""
    idx = torch.empty(len(q), k, dtype=torch.int64, device="cuda")
    dist = torch.empty(len(q), k, dtype=torch.float32, device="cuda")
    sq, sr = (q * q).sum(1), (r * r).sum(1)
    step = max(1, 400_000_000 // len(r))
    for s in range(0, len(q), step):
        e = min(len(q), s + step)
        d2 = torch.addmm(sr[None, :], q[s:e], r.T, alpha=-2.0).add_(sq[s:e, None]).clamp_(min=0.0)
        if self_rows:
            d2[torch.arange(e - s, device="cuda"), torch.arange(s, e, device="cuda")] = math.inf
        v, i = torch.topk(d2, k, dim=1, largest=False, sorted=True)
        idx[s:e], dist[s:e] = i, v.sqrt()
    return idx, dist


def _knn(x, rows, k):
    n = len(x)
    idx = torch.empty(n, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(n, k, dtype=torch.float32, device="cuda")
    for r in rows:
        c = x[r] - x[r].mean(0)  # the cluster's own frame keeps the float distances exact
        i, d = _search(c, c, k, True)
        idx[r], dist[r] = r[i].int(), d
    return idx, dist


def _graph(n, seed, k):
    x, y, rows = _mixture(n, seed, k)
    idx, dist = _knn(x, rows, k)
    return idx, dist, y


def _queries(n_ref, n_query, seed, k):
    x, y, rows = _mixture(n_ref, seed, k, extra=n_query)
    idx = torch.empty(n_query, k, dtype=torch.int32, device="cuda")
    dist = torch.empty(n_query, k, dtype=torch.float32, device="cuda")
    for r in rows:
        ref, q = r[r < n_ref], r[r >= n_ref]
        if len(q):
            near = ref if len(ref) >= k else torch.arange(n_ref, device="cuda")
            mid = x[near].mean(0)
            i, d = _search(x[q] - mid, x[near] - mid, k, False)
            idx[q - n_ref], dist[q - n_ref] = near[i].int(), d
    return y[:n_ref].double().cpu().numpy(), idx, dist


def _perplexity(k):
    return float(min(30, k // 3))


def _sizes(case):
    """Sizes of a batch's instances or a burst's requests, log-uniform over the case's range."""
    rng = np.random.default_rng(case["sizes"])
    count = case.get("instances") or case["requests"]
    s = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), count))
    return [int(v) for v in np.clip(np.round(s), case["lo"], case["hi"])]


def _inputs(case, seed):
    """The plain inputs of a case (no handle): what run() and exact() both start from."""
    kind = case["kind"]
    if kind in ("plan", "kl", "fit_device", "fit_host", "umap", "umap_spectral"):
        n, k = case["n"], case["k"]
        idx, dist, y = _graph(n, seed, k)
        if kind in ("fit_device", "fit_host") or (kind == "plan" and case["early"]):
            y = 0.3 * y  # early exaggeration works on a layout about this compact
        if kind in ("umap", "umap_spectral"):
            y = 0.2 * y
        return dict(idx=idx, dist=dist, y=y.cpu().numpy())
    if kind == "batch":
        graphs = [_graph(n, seed * 1000 + b, case["k"]) for b, n in enumerate(_sizes(case))]
        return dict(graphs=[(i, d, y.cpu().numpy()) for i, d, y in graphs])
    if kind == "pca":
        g = torch.Generator("cuda").manual_seed(int(seed))
        n, p = case["n"], case["p"]
        sd = 3.0 / torch.sqrt(torch.arange(1, p + 1, device="cuda", dtype=torch.float64))
        x = 2.0 + torch.randn(n, p, generator=g, device="cuda", dtype=torch.float64) * sd
        return dict(x=x.double().cpu().numpy() if case["double"] else x.float().cpu().numpy())
    if kind == "serve":
        sizes = _sizes(case)
        ref, idx, dist = _queries(case["n_ref"], sum(sizes), seed, case["k"])
        cut = np.cumsum(sizes)[:-1]
        return dict(ref=ref, requests=list(zip(np.split(idx.cpu().numpy(), cut), np.split(dist.cpu().numpy(), cut))))
    ref, idx, dist = _queries(case["n_ref"], case["n_query"], seed, case["k"])
    return dict(ref=ref, idx=idx.cpu().numpy(), dist=dist.cpu().numpy().astype(np.float64))


def prepare(case, seed):
    s = dict(_inputs(case, seed), case=case)
    kind = case["kind"]
    if kind in ("plan", "kl", "fit_device"):
        # the library takes the device KNN column-major: (k, n) row-major
        s["idx"], s["dist"] = s["idx"].T.contiguous(), s["dist"].T.contiguous()
    if kind in ("fit_host", "umap", "umap_spectral"):
        s["idx"], s["dist"] = s["idx"].cpu().numpy() + 1, s["dist"].cpu().numpy()  # R's 1-based rows
    if kind in ("plan", "kl"):
        s["plan"] = api.TsnePlan(s.pop("idx"), s.pop("dist"), case["n"], case["k"], _perplexity(case["k"]),
                                 init=s["y"])
    if kind == "batch":
        graphs = s.pop("graphs")
        s["batch"] = api.TsneBatch([(i.cpu().numpy() + 1, d.cpu().numpy()) for i, d, _ in graphs],
                                   perplexity=_perplexity(case["k"]), inits=[y for _, _, y in graphs])
    if kind == "serve":
        s["server"] = api.TransformServer(s["ref"])
        s["requests"] = [(i + 1, d) for i, d in s["requests"]]
    if kind == "transform":
        s["idx"] = s["idx"] + 1
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "plan":
        s["plan"].run(case["iters"], 12.0 if case["early"] else 1.0, case["n"] * TSNE_RATE)
        return s["plan"].layout()
    if kind == "kl":
        return s["plan"].kl()
    if kind == "fit_device":
        n = case["n"]
        plan = api.TsnePlan(s["idx"], s["dist"], n, case["k"], _perplexity(case["k"]), init=s["y"])
        plan.run(case["early_iters"], 12.0, n * TSNE_RATE)
        plan.run(case["iters"], 1.0, n * TSNE_RATE)
        out = plan.layout()
        plan.close()
        return out
    if kind == "fit_host":
        return api.tsne_knn(s["idx"], s["dist"], perplexity=_perplexity(case["k"]), Y_init=s["y"],
                            learning_rate=case["n"] * TSNE_RATE, early_exaggeration_iter=case["early_iters"],
                            n_iter=case["iters"]).layout
    if kind == "batch":
        s["batch"].iterate(case["iters"], 1.0, TSNE_RATE)
        return s["batch"].layouts()
    if kind == "umap":
        return api.umap_knn(s["idx"], s["dist"], init=s["y"], n_epochs=case["epochs"], learning_rate=UMAP_RATE).layout
    if kind == "umap_spectral":
        return api.umap_knn(s["idx"], s["dist"], n_epochs=case["epochs"], learning_rate=SPECTRAL_RATE).layout
    if kind == "pca":
        return api.tsne_pca_init(s["x"])
    if kind == "serve":
        ids = [s["server"].submit(i, d) for i, d in s["requests"]]
        return [s["server"].result(r)[0] for r in ids]
    return api.transform_tsne(s["ref"], dict(indices=s["idx"], distances=s["dist"]),
                              initialization="weighted" if case["weighted"] else "median").layout


# ---------------------------------------------------------------------------- work
def _tsne_work(n, k, iters):
    """One iteration reads P (8 bytes an entry, about 1.7 n k entries) and reads and writes the
    point state; an entry costs about 12 operations, the grid convolution 5 M^2 log2(M^2) a
    transform over six transforms of side M = 2 G."""
    nnz = 1.7 * n * k
    m = 2.0 * (256 if n < 20_000 else 512 if n < 100_000 else 1024)
    return iters * (8 * nnz + 56 * n), iters * (12 * nnz + 100 * n + 6 * 5 * m * m * math.log2(m * m))


def work(case):
    kind = case["kind"]
    if kind == "plan":
        b, f = _tsne_work(case["n"], case["k"], case["iters"])
    elif kind in ("fit_device", "fit_host"):
        n, k = case["n"], case["k"]
        b, f = _tsne_work(n, k, case["early_iters"] + case["iters"])
        b, f = b + 8 * n * k + 8 * 1.7 * n * k, f + 20 * 6.0 * n * k  # KNN in, P out; the bisection
    elif kind == "batch":
        parts = [_tsne_work(n, case["k"], case["iters"]) for n in _sizes(case)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind in ("umap", "umap_spectral"):
        n, k = case["n"], case["k"]
        edges = 1.5 * n * k
        b = 8 * n * k + 16 * n + 12 * edges
        f = case["epochs"] * edges * 0.3 * 6 * 25.0
        if kind == "umap_spectral":
            rounds = 30 if n >= 10_000 else 60
            f += rounds * (16 * edges + 8 * 9 * 4 * n)
            b += rounds * 16 * 8 * n
    elif kind == "pca":
        n, p = case["n"], case["p"]
        b, f = (8 if case["double"] else 4) * n * p + 8 * n, n * p * (p + 1.0) + 4.0 * n * p
    elif kind == "serve":
        q = sum(_sizes(case))
        b, f = q * (8 * case["k"] + 16) + 8 * case["n_ref"], 250.0 * q * (256 + case["k"]) * 12
    elif kind == "transform":
        q = case["n_query"]
        b, f = q * (12 * case["k"] + 16) + 16 * case["n_ref"], 250.0 * q * (case["n_ref"] + case["k"]) * 12
    else:
        n, nnz = case["n"], 1.7 * case["n"] * case["k"]
        b, f = 8 * nnz + 8 * n, 6.0 * n * n / 2 + 20 * nnz
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------- 64-bit values
def _row_p(dist, perplexity):
    """Perplexity bisection of the rows in 64 bits (tolerance 1e-5, at most 200 steps)."""
    d2 = dist.double() ** 2
    s = d2 - d2.min(1, keepdim=True).values
    n = len(s)
    beta = torch.ones(n, dtype=torch.float64, device=s.device)
    lo = torch.full_like(beta, -math.inf)
    hi = torch.full_like(beta, math.inf)
    out = torch.empty_like(s)
    live = torch.arange(n, device=s.device)
    flat = (d2.max(1).values - d2.min(1).values) <= 1.2e-7 * torch.clamp(d2.max(1).values, min=1.0)
    out[flat] = 1.0 / s.shape[1]
    live = live[~flat]
    target = math.log(perplexity)
    for it in range(200):
        if not len(live):
            break
        b = beta[live, None]
        p = torch.exp(-b * s[live])
        sp = p.sum(1)
        diff = beta[live] * (s[live] * p).sum(1) / sp + torch.log(sp) - target
        done = diff.abs() < 1e-5 if it < 199 else torch.ones_like(diff, dtype=torch.bool)
        out[live[done]] = p[done] / sp[done, None]
        live, diff = live[~done], diff[~done]
        up = diff > 0
        lo[live] = torch.where(up, beta[live], lo[live])
        hi[live] = torch.where(up, hi[live], beta[live])
        nb = 0.5 * (lo[live] + hi[live])
        nb = torch.where(torch.isinf(hi[live]), beta[live] * 2, nb)
        beta[live] = torch.where(torch.isinf(lo[live]), beta[live] * 0.5, nb)
    return out


def _joint_p(idx, dist, perplexity):
    """Symmetrised P as (rows, columns, values); the values sum to one."""
    n, k = idx.shape
    p = _row_p(dist, perplexity).ravel()
    i = torch.arange(n, device=idx.device).repeat_interleave(k)
    j = idx.long().ravel()
    key, inv = torch.unique(torch.cat([i * n + j, j * n + i]), return_inverse=True)
    v = torch.zeros(len(key), dtype=torch.float64, device=idx.device).index_add_(0, inv, torch.cat([p, p]))
    return key // n, key % n, v / v.sum()


def _grid_terms(y, grid):
    """Repulsion by bilinear splat, convolution on the zero-padded grid and bilinear gather."""
    n = len(y)
    lo, hi = y.min(0).values, y.max(0).values
    mid = 0.5 * (lo + hi)
    half = 0.55 * (hi - lo).max() + 1e-3
    h = 2 * half / (grid - 1)
    u = ((y - (mid - half)) / h).clamp(0, grid - 1)
    base = u.floor().clamp(max=grid - 2).long()
    f = u - base
    d = y - mid
    q = torch.stack([torch.ones(n, dtype=y.dtype, device=y.device), d[:, 0], d[:, 1]], 1)
    w, at = [], []
    for a in (0, 1):
        for b in (0, 1):
            w.append((f[:, 1] if a else 1 - f[:, 1]) * (f[:, 0] if b else 1 - f[:, 0]))
            at.append((base[:, 1] + a) * grid + base[:, 0] + b)
    ch = torch.zeros(grid * grid, 3, dtype=y.dtype, device=y.device)
    for ww, aa in zip(w, at):
        ch.index_add_(0, aa, ww[:, None] * q)
    o = torch.arange(2 * grid, device=y.device)
    o = torch.where(o < grid, o, o - 2 * grid).double()
    ker = 1 / (1 + h * h * (o[:, None] ** 2 + o[None, :] ** 2))
    ker[grid, :] = 0
    ker[:, grid] = 0
    ch = ch.T.reshape(3, grid, grid)
    spec = torch.fft.rfft2(ch, s=(2 * grid, 2 * grid))
    pot = torch.fft.irfft2(spec * torch.fft.rfft2(ker * ker), s=(2 * grid, 2 * grid))[:, :grid, :grid].reshape(3, -1)
    phi = torch.fft.irfft2(spec[0] * torch.fft.rfft2(ker), s=(2 * grid, 2 * grid))[:grid, :grid]
    z = (ch[0] * phi).sum() - n
    g = sum(ww[:, None] * pot[:, aa].T for ww, aa in zip(w, at))
    return -(d * g[:, :1] - g[:, 1:]) / z


class _Fit:
    """The optimizer's iterations in 64 bits."""

    def __init__(self, idx, dist, y, perplexity):
        self.i, self.j, self.p = _joint_p(idx, dist, perplexity)
        self.y = torch.as_tensor(y, dtype=torch.float64, device="cuda")
        self.gain = torch.ones_like(self.y)
        self.up = torch.zeros_like(self.y)
        n = len(self.y)
        self.grid = 256 if n < 20_000 else 512 if n < 100_000 else 1024

    def run(self, iters, exag, lr):
        step = 16_000_000
        for _ in range(iters):
            g = _grid_terms(self.y, self.grid)
            for s in range(0, len(self.p), step):
                i, j = self.i[s:s + step], self.j[s:s + step]
                d = self.y[i] - self.y[j]
                g.index_add_(0, i, d * (exag * self.p[s:s + step] / (1 + (d * d).sum(1)))[:, None])
            turn = torch.sign(self.up) != torch.sign(g)
            self.gain = torch.where(turn, self.gain + 0.2, self.gain * 0.8 + 0.01).clamp(min=0.01)
            self.up = 0.8 * self.up - lr * self.gain * g
            norm = self.up.norm(dim=1, keepdim=True)
            self.up = torch.where(norm > 5.0, self.up * (5.0 / norm.clamp(min=1e-30)), self.up)
            self.y = self.y - self.y.mean(0) + self.up
        return self

    def layout(self):
        return (self.y - self.y.mean(0)).cpu().numpy()

    def kl(self):
        n, z = len(self.y), 0.0
        for s in range(0, n, 2000):
            d2 = ((self.y[s:s + 2000, None, :] - self.y[None, :, :]) ** 2).sum(2)
            z += float((1 / (1 + d2)).sum())
        z -= n
        q = 1 / (1 + ((self.y[self.i] - self.y[self.j]) ** 2).sum(1)) / z
        return float((self.p * torch.log((self.p + 1e-9) / (q + 1e-9))).sum())


_U32 = 0xFFFFFFFF


def _mix(v):
    v = ((v ^ (v >> 16)) * 0x7FEB352D) & _U32
    v = ((v ^ (v >> 15)) * 0x846CA68B) & _U32
    v = v ^ (v >> 16)
    return torch.where(v == 0, torch.full_like(v, 0x6D2B79F5), v)


def _place(ref, idx, dist, weighted=False, first=None):
    """transform_tsne with its defaults in 64 bits. `first`: each query's number in its own call."""
    ref = torch.as_tensor(ref, device="cuda")
    idx = torch.as_tensor(idx, device="cuda").long()
    dist = torch.as_tensor(dist, device="cuda").double()
    n_ref, (nq, k) = len(ref), idx.shape
    p = _row_p(dist, 5.0)
    nb = ref[idx]
    if weighted:
        w = 1 / (dist + 1e-6)
        y = (w[:, :, None] * nb).sum(1) / w.sum(1, keepdim=True)
    else:
        v = nb.sort(1).values
        y = v[:, k // 2] if k & 1 else 0.5 * (v[:, k // 2] + v[:, k // 2 - 1])
    gain, up = torch.ones_like(y), torch.zeros_like(y)
    number = torch.arange(nq, device="cuda") if first is None else torch.as_tensor(first, device="cuda")
    salt = ((number + 1) * 0x9E3779B9) & _U32
    for it in range(250):
        if n_ref <= 4096:
            r = ref[None]
        else:
            s = _mix(((4 + 65537 * (it + 1)) & _U32) ^ salt)
            pick = torch.empty(256, nq, dtype=torch.int64, device="cuda")
            for m in range(256):
                s = s ^ ((s << 13) & _U32)
                s = s ^ (s >> 17)
                s = s ^ ((s << 5) & _U32)
                pick[m] = (s * n_ref) >> 32
            r = ref[pick.T]
        d = y[:, None, :] - r
        q = 1 / (1 + (d * d).sum(2))
        rep = ((q * q)[:, :, None] * d).sum(1) / q.sum(1, keepdim=True)
        d = y[:, None, :] - nb
        att = ((p / (1 + (d * d).sum(2)))[:, :, None] * d).sum(1)
        g = 1.5 * att - rep
        norm = g.norm(dim=1, keepdim=True)
        g = torch.where(norm > 0.25, g * 0.25 / (norm + 1e-12), g)
        gain = torch.where(torch.sign(up) != torch.sign(g), gain + 0.2, gain * 0.8 + 0.01).clamp(min=0.01)
        up = 0.8 * up - 0.1 * gain * g
        y = y + up
    return y.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("umap", "umap_spectral"):
        return None  # asynchronous updates: the result has no single 64-bit value
    s = _inputs(case, seed)
    if kind in ("plan", "kl", "fit_device", "fit_host"):
        lr = case["n"] * TSNE_RATE
        f = _Fit(s.pop("idx"), s.pop("dist"), s["y"], _perplexity(case["k"]))
        if kind == "kl":
            return f.kl()
        if kind == "plan":
            return f.run(case["iters"], 12.0 if case["early"] else 1.0, lr).layout()
        return f.run(case["early_iters"], 12.0, lr).run(case["iters"], 1.0, lr).layout()
    if kind == "batch":
        return [_Fit(i, d, y, _perplexity(case["k"])).run(case["iters"], 1.0, len(y) * TSNE_RATE).layout()
                for i, d, y in s["graphs"]]
    if kind == "pca":
        x = torch.as_tensor(s["x"], device="cuda").double()
        x = x - x.mean(0)
        v = torch.linalg.eigh(x.T @ x).eigenvectors[:, [-1, -2]]
        sc = x @ v
        top = sc.gather(0, sc.abs().argmax(0, keepdim=True))
        sc = sc * torch.where(top < 0, -1.0, 1.0)
        sc = sc - sc.mean(0)
        return (sc * (1e-4 / sc.std(0).max())).cpu().numpy()
    if kind == "serve":
        first = np.concatenate([np.arange(len(i)) for i, _ in s["requests"]])
        y = _place(s["ref"], np.concatenate([i for i, _ in s["requests"]]),
                   np.concatenate([d for _, d in s["requests"]]), first=first)
        return np.split(y, np.cumsum([len(i) for i, _ in s["requests"]])[:-1])
    return _place(s["ref"], s["idx"], s["dist"], case["weighted"])
