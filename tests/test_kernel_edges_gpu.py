"""Kernels and device functions launched alone. Rows of P, or of a UMAP graph, that end within a round of 2^31, the largest number of entries that is accepted: the
kernels that step over a row's entries, launched alone on arrays of 2^31 entries whose tail alone is filled.

Relabelling: exact. The others against FP64. Attraction: each lane sums at most two entries a row in FP32 and the warp's
sum has five levels, each term's factors and products are within 6 units of 2^-24: 2^-20 of the sum of magnitudes. KL:
the differences and d^2 are rounded to float, 2^-22 of log(1 + d^2) at most. Spectral: the weights are rounded to float once, 2^-23 allowed
for a tie; the products are FP64 sums of at most 300 terms, 2^-44.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from fastembedr_gb300 import _lib, build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))
ENTRIES, TAIL = 1 << 31, 1024
LAST = ENTRIES - 1  # the largest bound of a row


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    _lib.require_gpu()
    out = str(tmp_path_factory.mktemp("edges") / "kernel_edges.so")
    subprocess.run([build.nvcc(), "-std=c++17", *build.ARCH, "-O3", "-lineinfo", "-shared", "-Xcompiler", "-fPIC",
                    os.path.join(HERE, "kernel_edges.cu"), build.LIB, "-o", out], check=True)
    return C.CDLL(out)


def _rows(bounds):
    return np.array([[LAST - a, LAST - b] for a, b in bounds], np.int32)


# a whole round and part of one, a row within one round, rows beside each other on both sides of a multiple of 4
BOUNDS = [(500, 301), (301, 129), (129, 128), (128, 4), (4, 3), (3, 0), (600, 500), (601, 600)]


def test_relabel(lib):
    rows = _rows(BOUNDS)
    n = len(rows)
    rng = np.random.default_rng(1)
    delta = rng.permutation(n).astype(np.int32)
    col = rng.integers(0, n, TAIL).astype(np.int32)
    want = col.copy()
    for a, b in rows - (ENTRIES - TAIL):
        want[a:b] = delta[want[a:b]]
    assert lib.edge_relabel(rows.ctypes.data_as(C.c_void_p), n, col.ctypes.data_as(C.c_void_p), C.c_longlong(TAIL),
                            delta.ctypes.data_as(C.c_void_p)) == 0
    np.testing.assert_array_equal(col, want)


def test_attractive(lib):
    rows = _rows(BOUNDS)
    n = len(rows)
    rng = np.random.default_rng(2)
    col = rng.integers(0, n, TAIL).astype(np.int32)
    val = rng.uniform(0.0, 1.0, TAIL).astype(np.float32)
    y = rng.normal(size=(n, 2)).astype(np.float32)
    got = np.zeros((n, 2), np.float32)
    assert lib.edge_attractive(rows.ctypes.data_as(C.c_void_p), n, col.ctypes.data_as(C.c_void_p),
                               val.ctypes.data_as(C.c_void_p), C.c_longlong(TAIL), y.ctypes.data_as(C.c_void_p),
                               got.ctypes.data_as(C.c_void_p)) == 0
    y64 = y.astype(np.float64)
    for i, (a, b) in enumerate(rows - (ENTRIES - TAIL)):
        d = y64[i] - y64[col[a:b]]
        t = (val[a:b] / (1 + (d * d).sum(1)))[:, None] * d
        assert (np.abs(got[i] - t.sum(0)) <= 2.0 ** -20 * np.abs(t).sum(0)).all()


# contiguous rows up to the last entry: longer and shorter than a round of 32, a single entry, none
CONTIGUOUS = np.array([300, 140, 33, 33, 1, 0])


def _graph(seed):
    rng = np.random.default_rng(seed)
    bounds = (LAST - CONTIGUOUS).astype(np.int32)
    n = len(bounds) - 1
    return rng, bounds, n, rng.integers(0, n, TAIL).astype(np.int32), rng.uniform(0.01, 1.0, TAIL).astype(np.float32)


def test_kl(lib):
    rng, bounds, n, col, val = _graph(3)
    y = rng.normal(size=(n, 2)).astype(np.float32)
    z, got = 20.0, np.zeros(1)
    assert lib.edge_kl(bounds.ctypes.data_as(C.c_void_p), n, col.ctypes.data_as(C.c_void_p),
                       val.ctypes.data_as(C.c_void_p), C.c_longlong(TAIL), y.ctypes.data_as(C.c_void_p), C.c_double(z),
                       got.ctypes.data_as(C.c_void_p)) == 0
    want = size = 0.0
    for i in range(n):
        s = slice(bounds[i] - (ENTRIES - TAIL), bounds[i + 1] - (ENTRIES - TAIL))
        d = y[i].astype(np.float64) - y[col[s]]
        p = val[s].astype(np.float64)
        want += (p * np.log((p + 1e-9) / (1 / (1 + (d * d).sum(1)) / z + 1e-9))).sum()
        size += (p * np.log1p((d * d).sum(1))).sum()
    assert abs(got[0] - want) <= 2.0 ** -22 * size


def test_spectral(lib):
    rng, bounds, n, col, val = _graph(4)
    degree = rng.uniform(0.5, 2.0, n).astype(np.float32)
    x = rng.normal(size=(8, n))
    w, got = val.copy(), np.zeros((8, n))
    assert lib.edge_spectral(bounds.ctypes.data_as(C.c_void_p), n, col.ctypes.data_as(C.c_void_p),
                             w.ctypes.data_as(C.c_void_p), C.c_longlong(TAIL), degree.ctypes.data_as(C.c_void_p),
                             x.ctypes.data_as(C.c_void_p), 8, got.ctypes.data_as(C.c_void_p)) == 0
    for i in range(n):
        s = slice(bounds[i] - (ENTRIES - TAIL), bounds[i + 1] - (ENTRIES - TAIL))
        want = val[s] / np.sqrt(degree[i].astype(np.float64) * degree[col[s]].astype(np.float64))
        np.testing.assert_allclose(w[s], want, rtol=2.0 ** -23)
        t = w[s].astype(np.float64) * x[:, col[s]]
        assert (np.abs(got[:, i] - t.sum(1)) <= 2.0 ** -44 * np.abs(t).sum(1)).all()


# Bounds of the two-float functions, from their steps. exp: the polynomial, at most 1.5e-5, is rounded about five times in
# FP32 (2.2e-12), the table and the products to 2^-47. log: eight FP32 additions of low parts of at most 1.5e-6 |log2 x| +
# 3e-7 (7e-13 |log2 x| + 2e-13) and the rounding of |log2 x| 1.4e-6 (1.3e-13 |log2 x|).
def test_exp_two(lib):
    rng = np.random.default_rng(6)
    x = np.r_[-np.geomspace(1e-9, 50.0, 200001), -np.arange(0, 50, 0.0108304247, dtype=np.float64), 0.0]
    x = np.c_[x.astype(np.float32), np.zeros(len(x), np.float32)]
    x[:, 1] = x[:, 0] * rng.uniform(-2.0 ** -25, 2.0 ** -25, len(x))
    err = np.zeros(len(x))
    assert lib.edge_two_float(0, x.ctypes.data_as(C.c_void_p), len(x), err.ctypes.data_as(C.c_void_p)) == 0
    assert np.abs(err).max() <= 3e-12, (np.abs(err).max(), x[np.abs(err).argmax()])


def test_log_two(lib):
    rng = np.random.default_rng(7)
    x = np.r_[np.geomspace(1e-30, 1e30, 200001), np.linspace(0.5, 2.0, 100001), 2.0 ** np.arange(-100, 100)]
    x = np.c_[x.astype(np.float32), np.zeros(len(x), np.float32)]
    x[:, 1] = x[:, 0] * rng.uniform(-2.0 ** -25, 2.0 ** -25, len(x))
    err = np.zeros(len(x))
    assert lib.edge_two_float(1, x.ctypes.data_as(C.c_void_p), len(x), err.ctypes.data_as(C.c_void_p)) == 0
    bound = 1e-12 * (1.0 + np.abs(np.log2(x[:, 0].astype(np.float64))))
    assert (np.abs(err) <= bound).all(), (np.abs(err) / bound).max()


@pytest.mark.parametrize("exponent", [0, 1, 2, 7, 63, 124, 125, 128])
def test_reciprocal_is_correctly_rounded(lib, exponent):
    differ = C.c_ulonglong(1)
    assert lib.edge_reciprocal(exponent, C.byref(differ)) == 0
    assert differ.value == 0


# The sum over all pairs keeps FP64's digits though its terms are floats: they are correctly rounded, so their errors (a
# few 2^-25) have no common sign and average out over 10^8 pairs, as do those of the FP32 sums of 128 terms (rms
# 2e-7): 2e-7 / sqrt(4e5 sums) = 3e-10, three times that allowed.
@pytest.mark.parametrize("spread", [0.1, 30.0])
def test_normaliser(lib, spread):
    n = 10000
    y = (np.random.default_rng(8).standard_normal((n, 2)) * spread).astype(np.float32)
    got = C.c_double()
    assert lib.edge_z(y.ctypes.data_as(C.c_void_p), n, C.byref(got)) == 0
    y64 = y.astype(np.float64)
    want = sum((1 / (1 + ((y64[s:s + 500, None] - y64[None]) ** 2).sum(2))).sum() for s in range(0, n, 500)) - n
    assert got.value == pytest.approx(want, rel=1e-9)
